// Matrix products for many rows on pairs of SMs: y = x W^T in bfloat16 with 32-bit accumulation, finished in the epilogue.
//
// Two blocks of a cluster, on the two SMs of a pair, make one tile of 256 rows of x by 256 rows of W with
// tcgen05.mma.cta_group::2: each block stages 128 rows of either operand, so a 64-wide k step brings 32 KiB into an SM for
// the 4.2 MFLOP that a block of its own would need 48 KiB for (128 x 256), and L2 has a third less to deliver.  Per block: a
// ring of six stages (192 KiB) that runs on across tiles, the accumulator of 128 rows in 256 columns of tensor memory,
// twice, so that a tile is read back and stored while the next one is made.  Warp 0 copies (both blocks; bytes of both are
// counted by the leader's barrier), warp 1 of the leader issues the MMAs, warps 2 to 5 finish rows.  Clusters are persistent
// and take tiles c, c + clusters, ...
//
//   gated   W holds gate rows and up rows; the tile's 256 rows of W are 128 gate rows and the same features' 128 up rows,
//           fetched as four boxes of 64 rows, so either arrangement of the matrix can be read: gate rows in front of all up
//           rows, or groups of 64 in turn.  A thread finds gate and up of an output in columns j and 128 + j of its own row
//           and writes min(g, limit) * sigmoid(alpha * min(g, limit)) * (clamp(u) + up_shift), rounded once to bfloat16.  Expert
//           products divide to the last bit, as their kernel for tiles of 128 rows does (see quotient), dense ones as the
//           activation kernels for 16-bit rows do;
//   plain   the 32-bit sums are written as they are;
//   squared relu    max(sum, 0)^2 rounded once to bfloat16.
//
// With a tile table (see moe_plan) rows belong to experts: a tile is up to 256 rows of one expert's run, W that expert's
// matrix; rows behind the run's end are computed and not stored.
//
// What bounds it: with 2048 rows by W [24576, 4096] the tensor pipe is active in 78 % of the cycles (ncu), and the clock is what the
// power cap leaves of it, 1.70 GHz over one launch.  With the gate it takes 287 us on a cool GPU (1434 TFLOP/s; the library's product
// 305 us and its activation kernel 46) and 338 us on one that is at its power cap (library 325 + 48).  Expert products of 192 rows a
// run read W at 3.7 (gated) and 4.7 TB/s (plain) with the pipe active in 58 %: a quarter of each tile is rows that are not stored.
//
// Waits are bounded: a wait that runs out sets error code 7 in the flag, every role leaves its loop, both blocks meet
// at the cluster barriers and the tensor memory is freed.
#include "common.cuh"
#include "tcgen05.cuh"
#include "tma.cuh"

namespace {

constexpr int kRows = 128;           // rows of x per block (UMMA M is 256 over the pair)
constexpr int kCols = 256;           // rows of W per tile (UMMA N)
constexpr int kBox = 64;             // rows of W per copy
constexpr int kInner = 64;           // k per stage
constexpr int kRing = 6;
constexpr uint32_t kABytes = kRows * kInner * 2, kBBytes = kCols / 2 * kInner * 2, kStageBytes = kABytes + kBBytes;
constexpr int kThreads = 192;
constexpr int kPieceBytes = 32 * 128;      // what an epilogue warp hands to a bulk store: 128 bytes of each of its 32 rows
constexpr uint32_t kSharedBytes = kRing * kStageBytes + 4 * 2 * kPieceBytes + 1024;      // two pieces per epilogue warp

enum : int { FORM_PLAIN = 0, FORM_GATED = 1, FORM_SQUARED_RELU = 2 };

struct PairParams {
    const int* tiles;        // expert tiles (count first, then (expert, first row, rows) each), or null: all rows, one matrix
    int m;                   // rows of x without a tile table
    void* out;
    int out_cols;
    int col_tiles;
    int inner;
    int row_group;           // without a tile table: row tiles that are walked together for each column tile
    int interleave;          // gated: gate and up rows in turn, this many at a time (64); 0: all gate rows in front
    float limit, alpha, up_shift;
    int* error_flag;
};

__device__ __forceinline__ uint32_t pair_rank() {
    uint32_t rank;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    return rank;
}
__device__ __forceinline__ void pair_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// A shared-memory address of this block as the cluster sees the same place in block `rank`.
__device__ __forceinline__ uint32_t place_in(uint32_t address, uint32_t rank) {
    uint32_t remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(address), "r"(rank));
    return remote;
}
// A tile into this block's shared memory, its bytes counted by a barrier of either block of the pair.
__device__ __forceinline__ void load_pair(uint32_t dst, const CUtensorMap* map, uint32_t cluster_bar, int x, int y) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(dst), "l"(map), "r"(cluster_bar), "r"(x), "r"(y)
        : "memory");
}
__device__ __forceinline__ void mma_pair(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
        : "memory");
}
// Arrives on the barrier at this place in both blocks when all MMAs issued so far are complete.
__device__ __forceinline__ void commit_pair(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(bar), "h"((uint16_t)3) : "memory");
}
__device__ __forceinline__ void arrive_cluster(uint32_t cluster_bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}
// 64 columns of this warp's rows of the accumulator; the caller waits once for all loads that it has issued.
__device__ __forceinline__ void tmem_ask_64(uint32_t address, uint32_t (&r)[64]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x64.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32,%33,%34,%35,%36,%37,%38,%39,%40,%41,%42,%43,%44,%45,%46,%47,%48,%49,%50,%51,%52,%53,%54,%55,%56,%57,%58,%59,%60,%61,%62,%63}, [%64];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31]), "=r"(r[32]), "=r"(r[33]), "=r"(r[34]), "=r"(r[35]), "=r"(r[36]), "=r"(r[37]), "=r"(r[38]), "=r"(r[39]), "=r"(r[40]), "=r"(r[41]), "=r"(r[42]), "=r"(r[43]), "=r"(r[44]), "=r"(r[45]), "=r"(r[46]), "=r"(r[47]), "=r"(r[48]), "=r"(r[49]), "=r"(r[50]), "=r"(r[51]), "=r"(r[52]), "=r"(r[53]), "=r"(r[54]), "=r"(r[55]), "=r"(r[56]), "=r"(r[57]), "=r"(r[58]), "=r"(r[59]), "=r"(r[60]), "=r"(r[61]), "=r"(r[62]), "=r"(r[63])
        : "r"(address)
        : "memory");
}
// Both arrays are operands, so that nothing reads them before the wait.
__device__ __forceinline__ void tmem_wait(uint32_t (&r)[64]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 64; ++i) asm volatile("" : "+r"(r[i]));
}
__device__ __forceinline__ void tmem_wait(uint32_t (&r)[64], uint32_t (&q)[64]) {
    tmem_wait(r);
#pragma unroll
    for (int i = 0; i < 64; ++i) asm volatile("" : "+r"(q[i]));
}
// g / d for d >= 1: the product with the hardware's reciprocal (off by one unit in the last place) and one Newton step on the
// quotient, q + (g - d q) r (P. Markstein, IBM J. Res. Dev. 34, 1990), whose remainder a fused multiply-add leaves exact; where
// there is no remainder (an infinite divisor or gate) the product is the answer.  The hardware's approximate division is off by two
// units and gives 0 for divisors beyond 2^126, that is for gates between -87.3 and -88.7; the division operator branches, so that a
// thread's 128 divisions of a tile wait one for another: 16 experts of 512 over 1024,
// 160 rows each, plan and both products: 35 us with the approximate division, 38 this way, 56 with the operator.
__device__ __forceinline__ float quotient(float g, float d) {
    float r;
    asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(d));
    const float q = g * r, rest = fmaf(-d, q, g);
    return rest == rest ? fmaf(rest, r, q) : q;
}
// Bounded wait that also sees what the other block did before it arrived.
__device__ __forceinline__ bool wait_cluster(uint32_t bar, uint32_t parity) {
    for (uint32_t i = 0; i < tma::kWaitLimit; ++i) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done) : "r"(bar), "r"(parity) : "memory");
        if (done) return true;
    }
    return false;
}

// An epilogue warp's output of a tile, one piece of 128 bytes per row after the other.  Rows that all belong to the tile go through
// shared memory (128-byte swizzle, free of bank conflicts) and leave as one bulk store per piece; a warp whose rows end
// inside its 32 stores the rows that exist, 16 bytes at a time.
struct PieceStore {
    const CUtensorMap* map;
    uint32_t buffers;        // two pieces
    unsigned char* row_out;  // this lane's row of the output
    long long row_bytes;     // bytes of a row of the output
    int first_row;           // of the warp
    bool whole, present;     // all 32 rows belong to the tile; this lane's does
    int lane, turn;

    // words: this lane's 128 bytes; byte: where they begin in the row of the output; x: the same in elements
    __device__ __forceinline__ void put(const uint32_t (&words)[32], int byte, int x) {
        if (byte >= row_bytes) return;
        if (whole) {
            const uint32_t buffer = buffers + (turn & 1) * kPieceBytes;
            if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");      // the piece before the last has been read
            __syncwarp();
#pragma unroll
            for (int c = 0; c < 8; ++c)
                asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(buffer + lane * 128 + ((c ^ (lane & 7)) << 4)), "r"(words[4 * c]),
                             "r"(words[4 * c + 1]), "r"(words[4 * c + 2]), "r"(words[4 * c + 3]) : "memory");
            tma::fence_proxy_async();
            __syncwarp();
            if (lane == 0) {
                asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];"
                             ::"l"(map), "r"(buffer), "r"(x), "r"(first_row) : "memory");
                asm volatile("cp.async.bulk.commit_group;" ::: "memory");
            }
            ++turn;
        } else if (present) {
#pragma unroll
            for (int c = 0; c < 8; ++c)
                if (byte + 16 * (c + 1) <= row_bytes)
                    *reinterpret_cast<uint4*>(row_out + byte + 16 * c) = make_uint4(words[4 * c], words[4 * c + 1], words[4 * c + 2], words[4 * c + 3]);
        }
    }
    __device__ __forceinline__ void finish() const {      // nothing may be left in shared memory when the block leaves
        if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    }
};

// Tile t of the walk: its first row, how many rows are stored, its expert and its column tile.  Without a tile table the
// walk takes `row_group` row tiles through all column tiles before the next ones, so that these rows stay in L2 while W passes.
struct PairTile {
    int first_row, n_rows, expert, col_tile;
};
__device__ __forceinline__ PairTile tile_of(const PairParams& p, int t) {
    PairTile tile;
    if (p.tiles != nullptr) {
        const int* entry = p.tiles + 1 + 3 * (t / p.col_tiles);
        tile.expert = entry[0];
        tile.first_row = entry[1];
        tile.n_rows = entry[2];
        tile.col_tile = t % p.col_tiles;
        return tile;
    }
    const int row_tiles = (p.m + 2 * kRows - 1) / (2 * kRows);
    const int per_group = p.row_group * p.col_tiles, group = t / per_group, rest = t - group * per_group;
    const int in_group = min(p.row_group, row_tiles - group * p.row_group);
    const int row_tile = group * p.row_group + rest % in_group;
    tile.col_tile = rest / in_group;
    tile.expert = 0;
    tile.first_row = row_tile * 2 * kRows;
    tile.n_rows = min(2 * kRows, p.m - tile.first_row);
    return tile;
}

template <int FORM, bool EXACT>
__global__ void __launch_bounds__(kThreads) gemm_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w,
                                                             const __grid_constant__ CUtensorMap map_out, const PairParams p) {
    pdl_trigger();
    constexpr bool GATED = FORM == FORM_GATED;
    extern __shared__ unsigned char pair_shared[];
    __shared__ __align__(8) uint64_t full[kRing], empty[kRing], acc_full[2], acc_empty[2];
    __shared__ uint32_t tmem_slot;
    __shared__ int failed;
    const uint32_t ring = (tma::smem_u32(pair_shared) + 1023u) & ~1023u;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = pair_rank();
    const int cluster = blockIdx.x >> 1, clusters = gridDim.x >> 1;
    const int k_tiles = (p.inner + kInner - 1) / kInner;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kRing; ++s) {
            tma::mbar_init(tma::smem_u32(&full[s]), 1);
            tma::mbar_init(tma::smem_u32(&empty[s]), 1);
        }
        for (int b = 0; b < 2; ++b) {
            tma::mbar_init(tma::smem_u32(&acc_full[b]), 1);
            tma::mbar_init(tma::smem_u32(&acc_empty[b]), 8);      // one arrival per epilogue warp of either block
        }
        tma::mbar_fence_init();
        failed = 0;
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tma::smem_u32(&tmem_slot)), "r"(2 * kCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc5::fence_before();
    __syncthreads();
    pair_sync();                 // both blocks' barriers exist before either signals the other's
    tc5::fence_after();
    const uint32_t tmem = tmem_slot;
    pdl_wait();
    const int total = p.tiles != nullptr ? p.tiles[0] * p.col_tiles : (p.m + 2 * kRows - 1) / (2 * kRows) * p.col_tiles;

    if (warp == 0) {
        if (lane == 0) {
            bool ok = true;
            int step = 0;                                  // k steps issued so far, over all of this pair's tiles
            for (int t = cluster; t < total && ok; t += clusters) {
                const PairTile tile = tile_of(p, t);
                const int a_row = tile.first_row + (int)rank * kRows;
                // this block's 128 of the tile's 256 rows of W, as two boxes: gate rows in the leader and up rows in the other
                int w_row0, w_row1;
                if (GATED) {
                    const int feature = tile.col_tile * (kCols / 2);
                    w_row0 = tile.expert * 2 * p.out_cols + (p.interleave ? 2 * feature + (int)rank * kBox : feature + (int)rank * p.out_cols);
                    w_row1 = w_row0 + (p.interleave ? 2 * kBox : kBox);
                } else {
                    w_row0 = tile.expert * p.out_cols + tile.col_tile * kCols + (int)rank * (kCols / 2);
                    w_row1 = w_row0 + kBox;
                }
                for (int kt = 0; kt < k_tiles; ++kt, ++step) {
                    const int s = step % kRing;
                    if (step >= kRing) ok = tma::mbar_wait(tma::smem_u32(&empty[s]), ((step / kRing) - 1) & 1);
                    if (!ok) break;
                    const uint32_t stage = ring + s * kStageBytes;
                    if (rank == 0) tma::mbar_expect_tx(tma::smem_u32(&full[s]), 2 * kStageBytes);
                    const uint32_t bar = place_in(tma::smem_u32(&full[s]), 0);
                    load_pair(stage, &map_a, bar, kt * kInner, a_row);
                    load_pair(stage + kABytes, &map_w, bar, kt * kInner, w_row0);
                    load_pair(stage + kABytes + kBBytes / 2, &map_w, bar, kt * kInner, w_row1);
                }
            }
            // the leader's last commits signal this block's barriers: it may not leave before they have come
            for (int back = step < kRing ? step : kRing; back > 0 && ok; --back)
                ok = tma::mbar_wait(tma::smem_u32(&empty[(step - back) % kRing]), ((step - back) / kRing) & 1);
            if (!ok) failed = 1;
        }
    } else if (warp == 1) {
        if (lane == 0 && rank == 0) {
            const uint32_t idesc = tc5::instruction(2 * kRows, kCols, false);
            bool ok = true;
            int step = 0, turn = 0;                        // turn: this pair's tiles so far
            for (int t = cluster; t < total && ok; t += clusters, ++turn) {
                const int b = turn & 1;
                if (turn >= 2) ok = wait_cluster(tma::smem_u32(&acc_empty[b]), ((turn >> 1) - 1) & 1);
                if (!ok) break;
                tc5::fence_after();
                for (int kt = 0; kt < k_tiles; ++kt, ++step) {
                    const int s = step % kRing;
                    ok = tma::mbar_wait(tma::smem_u32(&full[s]), (step / kRing) & 1);
                    if (!ok) break;
                    tc5::fence_after();
                    const uint32_t stage = ring + s * kStageBytes;
#pragma unroll
                    for (int ks = 0; ks < kInner / 16; ++ks)
                        mma_pair(tmem + b * kCols, tc5::desc_k_major(stage + ks * 32, 1024u), tc5::desc_k_major(stage + kABytes + ks * 32, 1024u),
                                 idesc, (kt > 0 || ks > 0) ? 1u : 0u);
                    commit_pair(tma::smem_u32(&empty[s]));
                }
                if (ok) commit_pair(tma::smem_u32(&acc_full[b]));      // arrives when the tile's last MMA is complete
            }
            if (!ok) failed = 1;
        }
    } else {
        const int quarter = warp & 3;                    // the tensor-memory lanes this warp may read
        const int warp_row = (int)rank * kRows + quarter * 32;
        const bool bounded = p.limit < INFINITY;
        constexpr int kElement = FORM == FORM_PLAIN ? 4 : 2;
        PieceStore store;
        store.map = &map_out;
        store.buffers = ring + kRing * kStageBytes + quarter * 2 * kPieceBytes;
        store.row_bytes = (long long)p.out_cols * kElement;
        store.lane = lane;
        store.turn = 0;
        bool ok = true;
        int turn = 0;
        for (int t = cluster; t < total && ok; t += clusters, ++turn) {
            const int b = turn & 1;
            const PairTile tile = tile_of(p, t);
            const int col0 = tile.col_tile * (GATED ? kCols / 2 : kCols);
            store.first_row = tile.first_row + warp_row;
            store.whole = warp_row + 32 <= tile.n_rows;
            store.present = warp_row + lane < tile.n_rows;
            store.row_out = reinterpret_cast<unsigned char*>(p.out) + (size_t)(store.first_row + lane) * store.row_bytes;
            ok = tma::mbar_wait(tma::smem_u32(&acc_full[b]), (turn >> 1) & 1);
            if (!ok) {
                failed = 1;
                break;
            }
            tc5::fence_after();
            const uint32_t address = tmem + b * kCols + ((uint32_t)(quarter * 32) << 16);
            // A load from tensor memory comes back behind the MMAs that are queued already (the ring's six stages, 2 to 3 us), so
            // each wait is for 128 columns: with eight waits of 32 columns the read-back took longer than the next tile's
            // products and 2048 x 24576 x 4096 ran at 1261 TFLOP/s without storing anything, against 1513 without reading.
            for (int half = 0; half < 2 && warp_row < tile.n_rows; ++half) {
                uint32_t first[64], second[64];
                tmem_ask_64(address + (GATED ? half * 64 : half * 128), first);
                tmem_ask_64(address + (GATED ? kCols / 2 + half * 64 : half * 128 + 64), second);
                tmem_wait(first, second);
                if (GATED) {
                    uint32_t words[32];
#pragma unroll
                    for (int e = 0; e < 64; e += 2) {
                        float y[2];
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            float g = __uint_as_float(first[e + h]), u = __uint_as_float(second[e + h]);
                            if (bounded) {       // fminf would turn a NaN into the limit
                                g = fminf(g, p.limit);
                                u = fminf(fmaxf(u, -p.limit), p.limit);
                            }
                            const float below = 1.0f + __expf(-p.alpha * g);
                            y[h] = (EXACT ? quotient(g, below) : __fdividef(g, below)) * (u + p.up_shift);
                        }
                        words[e / 2] = tc5::pack2(y[0], y[1]);
                    }
                    store.put(words, (col0 + half * 64) * kElement, col0 + half * 64);
                } else if (FORM == FORM_SQUARED_RELU) {
#pragma unroll
                    for (int part = 0; part < 2; ++part) {
                        uint32_t words[32];
#pragma unroll
                        for (int e = 0; e < 64; e += 2) {
                            const float y0 = fmaxf(__uint_as_float(part ? second[e] : first[e]), 0.0f);
                            const float y1 = fmaxf(__uint_as_float(part ? second[e + 1] : first[e + 1]), 0.0f);
                            words[e / 2] = tc5::pack2(y0 * y0, y1 * y1);
                        }
                        const int column = col0 + half * 128 + part * 64;
                        store.put(words, column * kElement, column);
                    }
                } else {
#pragma unroll
                    for (int part = 0; part < 4; ++part) {
                        uint32_t words[32];
#pragma unroll
                        for (int e = 0; e < 32; ++e) words[e] = part & 2 ? second[(part & 1) * 32 + e] : first[(part & 1) * 32 + e];
                        const int column = col0 + half * 128 + part * 32;
                        store.put(words, column * kElement, column);
                    }
                }
            }
            // this half of the tensor memory may be overwritten by the tile after the next
            tc5::fence_before();
            __syncwarp();
            if (lane == 0) arrive_cluster(place_in(tma::smem_u32(&acc_empty[b]), 0));
        }
        store.finish();
    }
    __syncwarp();
    tc5::fence_before();
    __syncthreads();
    if (failed)                  // a wait ran out: copies that may still be in flight get time to land
        for (int i = 0; i < 200; ++i) __nanosleep(1000);
    pair_sync();                 // nobody signals a block that has left, and the pair frees its tensor memory together
    tc5::fence_after();
    if (failed && threadIdx.x == 0 && p.error_flag) atomicExch(p.error_flag, 7);
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * kCols));
}

// Tensor map of the output [rows, columns] (float or bfloat16) for pieces of 32 rows x 128 bytes; what lies outside is not written.
bool make_piece_map(CUtensorMap* map, void* pointer, uint64_t rows, uint64_t columns, bool wide) {
    tma::EncodeTiled encode = tma::encode_tiled();
    if (encode == nullptr) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)columns, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)columns * (wide ? 4 : 2)};
    const cuuint32_t box[2] = {wide ? 32u : 64u, 32u};
    const cuuint32_t ones[2] = {1, 1};
    return encode(map, wide ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, pointer, dims, strides, box, ones,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int FORM, bool EXACT>
int launch_pair(const CUtensorMap& map_a, const CUtensorMap& map_w, const CUtensorMap& map_out, const PairParams& p, long long most_tiles,
                cudaStream_t stream) {
    const size_t shared = kSharedBytes;
    if (int status = llm_raise_shared_limit((const void*)gemm_pair_kernel<FORM, EXACT>, shared, "gemm_pair")) return status;
    const int pairs = llm_sm_count() / 2;
    if (pairs < 1) {
        llm_set_error("gemm_pair: the device has no pair of SMs");
        return LLM_REFUSED;
    }
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3((unsigned)(2 * (most_tiles < pairs ? most_tiles : pairs)), 1, 1);
    config.blockDim = dim3(kThreads, 1, 1);
    config.dynamicSmemBytes = shared;
    config.stream = stream;
    cudaLaunchAttribute attribute[2];
    attribute[0].id = cudaLaunchAttributeClusterDimension;
    attribute[0].val.clusterDim.x = 2;
    attribute[0].val.clusterDim.y = 1;
    attribute[0].val.clusterDim.z = 1;
    attribute[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attribute[1].val.programmaticStreamSerializationAllowed = 1;
    config.attrs = attribute;
    config.numAttrs = llm_pdl_enabled() ? 2 : 1;
    const cudaError_t status = cudaLaunchKernelEx(&config, gemm_pair_kernel<FORM, EXACT>, map_a, map_w, map_out, p);
    if (status != cudaSuccess) {
        llm_set_error("gemm_pair launch: %s", cudaGetErrorString(status));
        return (int)status;
    }
    return llm_check_launch("gemm_pair");
}

int launch_form(int form, const void* a, int n_rows, const void* w, long long w_rows, PairParams p, long long row_tiles, cudaStream_t stream) {
    const bool gated = form == FORM_GATED;
    CUtensorMap map_a, map_w, map_out;
    if (!tma::make_map_bf16(&map_a, a, (uint64_t)n_rows, (uint64_t)p.inner, kRows) ||
        !tma::make_map_bf16(&map_w, w, (uint64_t)w_rows, (uint64_t)p.inner, kBox) ||
        !make_piece_map(&map_out, p.out, (uint64_t)n_rows, (uint64_t)p.out_cols, form == FORM_PLAIN)) {
        llm_set_error("gemm_pair: the tensor maps could not be made");
        return LLM_REFUSED;
    }
    const int per_tile = gated ? kCols / 2 : kCols;
    p.col_tiles = (p.out_cols + per_tile - 1) / per_tile;
    // row tiles whose rows of x (256 each) stay in L2 together while W passes: at most 32 MiB of them
    const long long tile_bytes = 2LL * kRows * p.inner * 2;
    const long long fit = (32LL << 20) / tile_bytes;
    p.row_group = (int)(fit < 1 ? 1 : fit > 16 ? 16 : fit);
    const long long most = row_tiles * p.col_tiles;
    if (gated && p.tiles != nullptr) return launch_pair<FORM_GATED, true>(map_a, map_w, map_out, p, most, stream);
    if (gated) return launch_pair<FORM_GATED, false>(map_a, map_w, map_out, p, most, stream);
    if (form == FORM_SQUARED_RELU) return launch_pair<FORM_SQUARED_RELU, true>(map_a, map_w, map_out, p, most, stream);
    return launch_pair<FORM_PLAIN, true>(map_a, map_w, map_out, p, most, stream);
}

}  // namespace

// `interleave`: rows of gate and up in turn (0: all gate rows in front); groups of 64 need a multiple of 64 features.
LLM_EXPORT int llm_gemm_pair_supports(int out_cols, int inner, int interleave) {
    return inner >= 64 && inner % 8 == 0 && out_cols > 0 && out_cols % 8 == 0 && (interleave == 0 || (interleave == kBox && out_cols % kBox == 0));
}

// out[m, features] = the gated activation of x[m, inner] W^T, W [2 features, inner] bfloat16; bfloat16 out.
LLM_EXPORT int llm_gemm_pair_gated(const void* x, const void* w, void* out, int m, int features, int inner, int interleave, float limit,
                                   float alpha, float up_shift, int* error_flag, cudaStream_t stream) {
    if (m <= 0) return LLM_OK;
    if (!llm_gemm_pair_supports(features, inner, interleave) || !aligned16(x) || !aligned16(w) || !aligned16(out)) {
        llm_set_error("gemm_pair_gated: %d features over an inner size of %d (rows in turn: %d) are not supported", features, inner, interleave);
        return LLM_REFUSED;
    }
    PairParams p = {};
    p.m = m;
    p.out = out;
    p.out_cols = features;
    p.inner = inner;
    p.interleave = interleave;
    p.limit = limit;
    p.alpha = alpha;
    p.up_shift = up_shift;
    p.error_flag = error_flag;
    return launch_form(FORM_GATED, x, m, w, 2LL * features, p, (m + 2 * kRows - 1) / (2 * kRows), stream);
}

// The expert products of moe_grouped_tcgen05.cu on pairs of SMs; `tiles` holds tiles of up to 256 rows.  Arguments as there.
LLM_EXPORT int llm_moe_grouped_pair(const void* a, int n_rows, const void* w, int experts, const int* tiles, void* out, int out_cols,
                                    int inner, int max_tiles, int form, float limit, float alpha, float up_shift, int* error_flag,
                                    cudaStream_t stream) {
    if (max_tiles <= 0 || n_rows <= 0) return LLM_OK;
    if (!llm_gemm_pair_supports(out_cols, inner, 0) || !aligned16(a) || !aligned16(w) || !aligned16(out)) {
        llm_set_error("moe_grouped_pair: %d output columns over an inner size of %d are not supported (both multiples of 8, "
                      "16-byte aligned operands)", out_cols, inner);
        return LLM_REFUSED;
    }
    PairParams p = {};
    p.tiles = tiles;
    p.m = n_rows;
    p.out = out;
    p.out_cols = out_cols;
    p.inner = inner;
    p.limit = limit;
    p.alpha = alpha;
    p.up_shift = up_shift;
    p.error_flag = error_flag;
    return launch_form(form, a, n_rows, w, (long long)experts * (form == FORM_GATED ? 2 : 1) * out_cols, p, max_tiles, stream);
}
