// Gated linear attention: the recurrence over a step's tokens, with its state in 32-bit per request.
//
// Per head, with key channels i < dim and value channels j < vdim:
//     alpha_t[i] = sigmoid(z_t[i] + b[i]) ^ (1 / tau)         = exp(-softplus(-(z + b)) / tau), formed in 32-bit
//     S_t[i][j]  = alpha_t[i] * S_(t-1)[i][j] + k_t[i] * v_t[j]
//     o_t[j]     = sum_i S_t[i][j] * q_t[i] * q_scale
//     out_t[j]   = o_t[j] / sqrt(mean_j(o_t^2) + eps) * weight[j] * silu(g_t[j])
// q, k, v and g are column ranges of one packed projection row; z is a projection of its own, kept in 32-bit (the
// decay is the one quantity here whose error compounds from token to token).  The state of a
// sequence lives in its slot of `state` [slots, heads, dim, vdim] (float32): it is read when the block starts on the
// sequence's tokens of this step and written back behind the last of them, so a prompt may arrive in portions of any
// size and single decoded tokens continue it.  A slot that a new request takes over is zeroed by the cache manager.
//
// One block per (sequence, head).  A thread owns `R` rows of one column of S in registers; `P` such row partitions
// cover dim.  Tokens are taken sixteen at a time: (1) the block stages their q, k, alpha and v in shared memory, the decay
// and everything else that enters the recurrence in 32-bit; (2) every thread walks the sixteen tokens on its registers
// and leaves its partial o; (3) the warps add the partitions' parts in a fixed order, normalise, gate and store.  The
// order of every sum depends on the sizes alone, so a token's result does not depend on how the prompt was cut or on
// what else is in the batch.  (In bfloat16 steps with heads of 64 key channels the kernels further down run: there the states have the
// same bits whichever of them made them in one pass, but o's sums have one order in steps of single tokens alone and another in steps with portions.)
//
// Long portions can also be walked segment by segment in parallel (`llm_gla_recurrent` with a segment length): pass A
// runs every segment but the last from a zero state and leaves its end state and the product of its decays; a scan adds
// them up, S_in(k+1) = D_k S_in(k) + S_local(k), which gives every segment the state it starts from; pass C runs the
// segments again from those states and writes the outputs.  Twice the arithmetic, all of it still 32-bit, on as many
// blocks as there are segments; sums are then grouped by segment, so results agree with the one-pass form to rounding,
// not bit for bit (the 32-bit path keeps the one-pass form).
#include "common.cuh"
#include "tcgen05.cuh"      // two-wide 32-bit arithmetic

#define GLA_TOKENS 16

struct GlaArgs {
    const void* proj;       // [N, row_width]
    int row_width, q_offset, k_offset, v_offset, g_offset;
    const float* z;         // [N, heads * dim], 32-bit in either path
    const float* z_bias;    // [heads * dim] or null
    const void* weight;     // [vdim] norm weight
    float* state;           // [slots, heads, dim, vdim]
    const int* state_slots; // [S]
    const int* q_start;     // [S + 1]
    void* out;              // [N, heads * vdim]
    int heads, dim, vdim, partitions, padded_dim, column_threads;
    float inverse_tau, q_scale, eps;
    int segment, max_segments;   // segmented form: tokens per segment, segments the scratch has room for per sequence
    float* segment_state;        // [S, max_segments, heads, dim, vdim]
    float* segment_decay;        // [S, max_segments, heads, dim]
};

// MODE 0: a sequence's tokens in one pass, from and into its state slot.  1: pass A of the segmented form.  3: pass C.
enum : int { GLA_ONE_PASS = 0, GLA_LOCAL = 1, GLA_OUTPUT = 3 };

// R = 128 comes with 256 threads, where a thread's 128 rows of state fit its registers, and, for sizes nothing else
// takes, with 512 (R given as 129), where they spill: slow, but every size up to 256 x 256 then runs.
template <typename T, typename W, int RR, int MODE>
__global__ void __launch_bounds__(RR == 128 ? 256 : 512, RR <= 16 ? 2 : 1) gla_recurrent_kernel(GlaArgs a) {
    constexpr int R = RR == 129 ? 128 : RR;
    pdl_trigger();
    pdl_wait();
    extern __shared__ float4 gla_shared_raw[];
    float* shared = reinterpret_cast<float*>(gla_shared_raw);
    const int seq = blockIdx.x, head = blockIdx.y;
    int begin = a.q_start[seq], end = a.q_start[seq + 1];
    if (begin >= end) return;
    bool last_segment = true;
    size_t segment_index = 0;
    if (MODE != GLA_ONE_PASS) {
        const int segments = (end - begin + a.segment - 1) / a.segment;
        const int segment = blockIdx.z;
        if (segment >= segments) return;
        last_segment = segment == segments - 1;
        if (MODE == GLA_LOCAL && last_segment) return;      // nobody needs the state a zero start leaves behind the last one
        begin += segment * a.segment;
        end = min(end, begin + a.segment);
        segment_index = ((size_t)seq * a.max_segments + segment) * a.heads + head;
    }
    const int dim = a.dim, vdim = a.vdim, padded = a.padded_dim;
    float* q_s = shared;                                   // [GLA_TOKENS][padded]
    float* k_s = q_s + GLA_TOKENS * padded;
    float* alpha_s = k_s + GLA_TOKENS * padded;
    float* v_s = alpha_s + GLA_TOKENS * padded;            // [GLA_TOKENS][vdim]
    float* part_s = v_s + GLA_TOKENS * vdim;               // [partitions][GLA_TOKENS][vdim]
    const int column = threadIdx.x % a.column_threads, partition = threadIdx.x / a.column_threads;
    const int row0 = partition * R;
    const bool owner = column < vdim && partition < a.partitions;
    const T* proj = (const T*)a.proj;
    const float* z = a.z;

    float S[R];
    float decay[MODE == GLA_LOCAL ? R : 1];      // pass A: the product of the segment's decays, row by row
    float* state = a.state + ((size_t)a.state_slots[seq] * a.heads + head) * dim * vdim;
    float* segment_state = a.segment_state + segment_index * dim * vdim;
    const float* source = MODE == GLA_OUTPUT ? segment_state : state;
#pragma unroll
    for (int i = 0; i < R; ++i) {
        S[i] = (MODE != GLA_LOCAL && owner && row0 + i < dim) ? source[(size_t)(row0 + i) * vdim + column] : 0.0f;
        if (MODE == GLA_LOCAL) decay[i] = 1.0f;
    }

    for (int first = begin; first < end; first += GLA_TOKENS) {
        const int count = min(GLA_TOKENS, end - first);
        __syncthreads();      // the parts of the tokens before have been read
        for (int e = threadIdx.x; e < count * padded; e += blockDim.x) {
            const int t = e / padded, i = e % padded;
            float qv = 0.0f, kv = 0.0f, alpha = 0.0f;
            if (i < dim) {
                const T* row = proj + (size_t)(first + t) * a.row_width;
                qv = Num<T>::load(row + a.q_offset + head * dim + i) * a.q_scale;
                kv = Num<T>::load(row + a.k_offset + head * dim + i);
                float zz = z[(size_t)(first + t) * a.heads * dim + head * dim + i];
                if (a.z_bias) zz += a.z_bias[head * dim + i];
                // log sigmoid(zz) = -softplus(-zz), stable on both sides
                const float log_sigmoid = zz >= 0.0f ? -log1pf(expf(-zz)) : zz - log1pf(expf(zz));
                alpha = expf(log_sigmoid * a.inverse_tau);
            }
            q_s[e] = qv;
            k_s[e] = kv;
            alpha_s[e] = alpha;
        }
        for (int e = threadIdx.x; e < count * vdim; e += blockDim.x) {
            const int t = e / vdim, j = e % vdim;
            v_s[e] = Num<T>::load(proj + (size_t)(first + t) * a.row_width + a.v_offset + head * vdim + j);
        }
        __syncthreads();
        if (owner) {
            for (int t = 0; t < count; ++t) {
                const float vj = v_s[t * vdim + column];
                const float4* q4 = reinterpret_cast<const float4*>(q_s + t * padded + row0);
                const float4* k4 = reinterpret_cast<const float4*>(k_s + t * padded + row0);
                const float4* a4 = reinterpret_cast<const float4*>(alpha_s + t * padded + row0);
                float o = 0.0f;
#pragma unroll
                for (int i = 0; i < R / 4; ++i) {
                    const float4 qq = q4[i], kk = k4[i], aa = a4[i];
                    S[4 * i + 0] = fmaf(aa.x, S[4 * i + 0], kk.x * vj);
                    S[4 * i + 1] = fmaf(aa.y, S[4 * i + 1], kk.y * vj);
                    S[4 * i + 2] = fmaf(aa.z, S[4 * i + 2], kk.z * vj);
                    S[4 * i + 3] = fmaf(aa.w, S[4 * i + 3], kk.w * vj);
                    if (MODE == GLA_LOCAL) {
                        decay[4 * i + 0] *= aa.x;
                        decay[4 * i + 1] *= aa.y;
                        decay[4 * i + 2] *= aa.z;
                        decay[4 * i + 3] *= aa.w;
                    } else {
                        o = fmaf(S[4 * i + 0], qq.x, o);
                        o = fmaf(S[4 * i + 1], qq.y, o);
                        o = fmaf(S[4 * i + 2], qq.z, o);
                        o = fmaf(S[4 * i + 3], qq.w, o);
                    }
                }
                if (MODE != GLA_LOCAL) part_s[((size_t)partition * GLA_TOKENS + t) * vdim + column] = o;
            }
        }
        if (MODE == GLA_LOCAL) continue;
        __syncthreads();
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
        for (int t = warp; t < count; t += warps) {
            float sum_squares = 0.0f;
            for (int j = lane; j < vdim; j += 32) {
                float o = 0.0f;
                for (int p = 0; p < a.partitions; ++p) o += part_s[((size_t)p * GLA_TOKENS + t) * vdim + j];
                part_s[(size_t)t * vdim + j] = o;      // partition 0's place: each element is read and written by one lane
                sum_squares += o * o;
            }
            const float inverse = rsqrtf(warp_sum(sum_squares) / (float)vdim + a.eps);
            const T* g_row = proj + (size_t)(first + t) * a.row_width + a.g_offset + head * vdim;
            T* dst = (T*)a.out + (size_t)(first + t) * a.heads * vdim + head * vdim;
            for (int j = lane; j < vdim; j += 32) {
                const float g = Num<T>::load(g_row + j);
                const float gate = g / (1.0f + expf(-g));
                Num<T>::store(dst + j, part_s[(size_t)t * vdim + j] * inverse * Num<W>::load((const W*)a.weight + j) * gate);
            }
        }
    }
    if (owner && (MODE == GLA_LOCAL || last_segment)) {
        float* target = MODE == GLA_LOCAL ? segment_state : state;
#pragma unroll
        for (int i = 0; i < R; ++i)
            if (row0 + i < dim) target[(size_t)(row0 + i) * vdim + column] = S[i];
        if (MODE == GLA_LOCAL && column == 0) {
#pragma unroll
            for (int i = 0; i < R; ++i)
                if (row0 + i < dim) a.segment_decay[segment_index * dim + row0 + i] = decay[i];
        }
    }
}

// The same passes for bfloat16 steps and heads of 64 key channels, where a thread owns a tile of S: 8 rows of 8 columns, so that what
// it reads of shared memory for a token (q, k and alpha of its rows, v of its columns: eight 16-byte loads) serves 192
// multiply-adds, made two at a time (fma.rn.f32x2 over pairs of rows).  A warp holds 32 columns of S: lane = row group + 8 * column
// group, row group r has rows 4 r .. 4 r + 3 and 32 + 4 r .. 32 + 4 r + 3 (so that the eight groups of a load are 128 contiguous
// bytes), and the row groups' parts of o are added by seven shuffles, each of which halves the columns that a lane still holds.
// What bounds the kernel above for long portions is its staging: a thread's loads of a batch of tokens wait for one another (up to
// 16 in a row).  Here all of a batch is asked for at once, 16 bytes at a time.  2048 tokens of 32 heads of 64 / 128, us, the
// kernel above / this: states of the segments 153 / 73, outputs 232 / 133 (tiles with loads one after the other: 148 and 254; outputs
// with the gates read at a batch's end: 156; without two tokens in flight: 142, which would make the states' pass 82).  The sizes of
// this layer in the package are 64 / 128; a tile per thread of heads of 128 key channels would take other registers and was not
// built, so they stay with the kernel above.
constexpr int kTileDim = 64;

// Eight bfloat16 numbers, times `scale`, as 32-bit numbers in shared memory.
__device__ __forceinline__ void spread8(const float4& raw, float scale, float* dst) {
    const __nv_bfloat162* pairs = reinterpret_cast<const __nv_bfloat162*>(&raw);
    float v[8];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const float2 both = __bfloat1622float2(pairs[c]);
        v[2 * c] = both.x * scale;
        v[2 * c + 1] = both.y * scale;
    }
    *reinterpret_cast<float4*>(dst) = make_float4(v[0], v[1], v[2], v[3]);
    *reinterpret_cast<float4*>(dst + 4) = make_float4(v[4], v[5], v[6], v[7]);
}

template <typename W, int VDIM, int MODE>
__global__ void __launch_bounds__(VDIM) gla_tiles_kernel(GlaArgs a) {
    pdl_trigger();
    pdl_wait();
    typedef __nv_bfloat16 T;
    extern __shared__ float4 gla_shared_raw[];
    float* shared = reinterpret_cast<float*>(gla_shared_raw);
    const int seq = blockIdx.x, head = blockIdx.y;
    int begin = a.q_start[seq], end = a.q_start[seq + 1];
    if (begin >= end) return;
    bool last_segment = true;
    size_t segment_index = 0;
    if (MODE != GLA_ONE_PASS) {
        const int segments = (end - begin + a.segment - 1) / a.segment;
        const int segment = blockIdx.z;
        if (segment >= segments) return;
        last_segment = segment == segments - 1;
        if (MODE == GLA_LOCAL && last_segment) return;      // nobody needs the state a zero start leaves behind the last one
        begin += segment * a.segment;
        end = min(end, begin + a.segment);
        segment_index = ((size_t)seq * a.max_segments + segment) * a.heads + head;
    }
    float* q_s = shared;                                   // [GLA_TOKENS][64]
    float* k_s = q_s + GLA_TOKENS * kTileDim;
    float* alpha_s = k_s + GLA_TOKENS * kTileDim;
    float* v_s = alpha_s + GLA_TOKENS * kTileDim;          // [GLA_TOKENS][VDIM]
    float* o_s = v_s + GLA_TOKENS * VDIM;                  // [GLA_TOKENS][VDIM]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int kWarps = VDIM / 32;
    const int row_group = lane & 7, column0 = warp * 32 + (lane >> 3) * 8;
    const T* proj = (const T*)a.proj;

    uint64_t S[4][8];                                       // [pair of rows][column]
    uint64_t decay[MODE == GLA_LOCAL ? 4 : 1];               // pass A: the product of the segment's decays
    float* state = a.state + ((size_t)a.state_slots[seq] * a.heads + head) * kTileDim * VDIM;
    float* segment_state = a.segment_state + segment_index * kTileDim * VDIM;
    const float* source = MODE == GLA_OUTPUT ? segment_state : state;
    auto row_of = [&](int pair) { return 4 * row_group + (pair >> 1) * 32 + (pair & 1) * 2; };
#pragma unroll
    for (int pair = 0; pair < 4; ++pair) {
        if (MODE == GLA_LOCAL) {
            decay[pair] = tc5::pair_of(1.0f, 1.0f);
#pragma unroll
            for (int c = 0; c < 8; ++c) S[pair][c] = 0;
        } else {
            const float* first = source + (size_t)row_of(pair) * VDIM + column0;
#pragma unroll
            for (int c = 0; c < 8; c += 4) {
                const float4 low = *reinterpret_cast<const float4*>(first + c), high = *reinterpret_cast<const float4*>(first + VDIM + c);
                S[pair][c] = tc5::pair_of(low.x, high.x);
                S[pair][c + 1] = tc5::pair_of(low.y, high.y);
                S[pair][c + 2] = tc5::pair_of(low.z, high.z);
                S[pair][c + 3] = tc5::pair_of(low.w, high.w);
            }
        }
    }
    float weights[VDIM / 32];                        // of the norm, for the columns of a token that this lane finishes
#pragma unroll
    for (int j = 0; j < VDIM / 32; ++j) weights[j] = Num<W>::load((const W*)a.weight + lane * (VDIM / 32) + j);
    const int my_column = column0 + row_group;      // the one of its eight that a lane holds when the row groups' parts have been added

    for (int first = begin; first < end; first += GLA_TOKENS) {
        const int count = min(GLA_TOKENS, end - first);
        __syncthreads();      // what the tokens before left in shared memory has been read
        // Everything a batch of tokens needs is asked for before the first of it is used, 16 bytes at a time.
        constexpr int kNarrow = GLA_TOKENS * kTileDim / 8, kWide = GLA_TOKENS * kTileDim / 4, kValues = GLA_TOKENS * VDIM / 8;
        constexpr int kNarrowEach = (kNarrow + VDIM - 1) / VDIM, kWideEach = (kWide + VDIM - 1) / VDIM, kValuesEach = (kValues + VDIM - 1) / VDIM;
        float4 q_raw[kNarrowEach], k_raw[kNarrowEach], z_raw[kWideEach], v_raw[kValuesEach];
#pragma unroll
        for (int u = 0; u < kNarrowEach; ++u) {
            const int e = threadIdx.x + u * VDIM, t = e / (kTileDim / 8), i = e % (kTileDim / 8) * 8;
            if (e < kNarrow && t < count) {
                const T* row = proj + (size_t)(first + t) * a.row_width + head * kTileDim + i;
                if (MODE != GLA_LOCAL) q_raw[u] = *reinterpret_cast<const float4*>(row + a.q_offset);
                k_raw[u] = *reinterpret_cast<const float4*>(row + a.k_offset);
            }
        }
#pragma unroll
        for (int u = 0; u < kWideEach; ++u) {
            const int e = threadIdx.x + u * VDIM, t = e / (kTileDim / 4), i = e % (kTileDim / 4) * 4;
            if (e < kWide && t < count) z_raw[u] = *reinterpret_cast<const float4*>(a.z + ((size_t)(first + t) * a.heads + head) * kTileDim + i);
        }
#pragma unroll
        for (int u = 0; u < kValuesEach; ++u) {
            const int e = threadIdx.x + u * VDIM, t = e / (VDIM / 8), j = e % (VDIM / 8) * 8;
            if (t < count) v_raw[u] = *reinterpret_cast<const float4*>(proj + (size_t)(first + t) * a.row_width + a.v_offset + head * VDIM + j);
        }
        // (the gates of the tokens that this warp will finish, too)
        constexpr int kEach = VDIM / 32, kMine = GLA_TOKENS / kWarps;      // neighbouring columns of a lane, tokens of a warp
        uint32_t g_raw[MODE == GLA_LOCAL ? 1 : kMine][kEach / 2];
        if (MODE != GLA_LOCAL) {
#pragma unroll
            for (int u = 0; u < kMine; ++u) {
                const int t = warp + u * kWarps;
                const uint32_t* g_row = reinterpret_cast<const uint32_t*>(proj + (size_t)(first + t) * a.row_width + a.g_offset + head * VDIM + lane * kEach);
#pragma unroll
                for (int j = 0; j < kEach / 2; ++j) g_raw[u][j] = t < count ? g_row[j] : 0u;
            }
        }
#pragma unroll
        for (int u = 0; u < kNarrowEach; ++u) {
            const int e = threadIdx.x + u * VDIM;
            if (e < kNarrow && e / (kTileDim / 8) < count) {
                if (MODE != GLA_LOCAL) spread8(q_raw[u], a.q_scale, q_s + e * 8);
                spread8(k_raw[u], 1.0f, k_s + e * 8);
            }
        }
#pragma unroll
        for (int u = 0; u < kWideEach; ++u) {
            const int e = threadIdx.x + u * VDIM, i = e % (kTileDim / 4) * 4;
            if (e < kWide && e / (kTileDim / 4) < count) {
                float zz[4] = {z_raw[u].x, z_raw[u].y, z_raw[u].z, z_raw[u].w};
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    if (a.z_bias) zz[c] += a.z_bias[head * kTileDim + i + c];
                    // log sigmoid(zz) = -softplus(-zz), stable on both sides
                    const float log_sigmoid = zz[c] >= 0.0f ? -log1pf(expf(-zz[c])) : zz[c] - log1pf(expf(zz[c]));
                    zz[c] = expf(log_sigmoid * a.inverse_tau);
                }
                *reinterpret_cast<float4*>(alpha_s + e * 4) = make_float4(zz[0], zz[1], zz[2], zz[3]);
            }
        }
#pragma unroll
        for (int u = 0; u < kValuesEach; ++u) {
            const int e = threadIdx.x + u * VDIM;
            if (e / (VDIM / 8) < count) spread8(v_raw[u], 1.0f, v_s + e * 8);
        }
        __syncthreads();
#pragma unroll(MODE == GLA_LOCAL ? 1 : 2)
        for (int t = 0; t < count; ++t) {
            const int at = t * kTileDim + 4 * row_group;
            const ulonglong2 k_low = *reinterpret_cast<const ulonglong2*>(k_s + at), k_high = *reinterpret_cast<const ulonglong2*>(k_s + at + 32);
            const ulonglong2 a_low = *reinterpret_cast<const ulonglong2*>(alpha_s + at), a_high = *reinterpret_cast<const ulonglong2*>(alpha_s + at + 32);
            const uint64_t k[4] = {k_low.x, k_low.y, k_high.x, k_high.y}, alpha[4] = {a_low.x, a_low.y, a_high.x, a_high.y};
            const float4 v_low = *reinterpret_cast<const float4*>(v_s + t * VDIM + column0), v_high = *reinterpret_cast<const float4*>(v_s + t * VDIM + column0 + 4);
            const float v[8] = {v_low.x, v_low.y, v_low.z, v_low.w, v_high.x, v_high.y, v_high.z, v_high.w};
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                const uint64_t vv = tc5::pair_of(v[c], v[c]);
#pragma unroll
                for (int pair = 0; pair < 4; ++pair) S[pair][c] = tc5::fma_pair(alpha[pair], S[pair][c], tc5::mul_pair(k[pair], vv));
            }
            if (MODE == GLA_LOCAL) {
#pragma unroll
                for (int pair = 0; pair < 4; ++pair) decay[pair] = tc5::mul_pair(decay[pair], alpha[pair]);
                continue;
            }
            const ulonglong2 q_low = *reinterpret_cast<const ulonglong2*>(q_s + at), q_high = *reinterpret_cast<const ulonglong2*>(q_s + at + 32);
            const uint64_t q[4] = {q_low.x, q_low.y, q_high.x, q_high.y};
            float o[8];
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                uint64_t sum = tc5::mul_pair(S[0][c], q[0]);
#pragma unroll
                for (int pair = 1; pair < 4; ++pair) sum = tc5::fma_pair(S[pair][c], q[pair], sum);
                float low, high;
                tc5::halves_of(sum, low, high);
                o[c] = low + high;
            }
#pragma unroll
            for (int held = 4; held > 0; held >>= 1) {      // of 2 * held columns a lane keeps the half that its row group names
                const bool upper = row_group & held;
#pragma unroll
                for (int c = 0; c < held; ++c) {
                    const float mine = upper ? o[c + held] : o[c], other = upper ? o[c] : o[c + held];
                    o[c] = mine + __shfl_xor_sync(0xffffffffu, other, held);
                }
            }
            o_s[t * VDIM + my_column] = o[0];
        }
        if (MODE == GLA_LOCAL) continue;
        __syncthreads();
#pragma unroll
        for (int u = 0; u < kMine; ++u) {
            const int t = warp + u * kWarps;
            if (t >= count) break;
            T* dst = (T*)a.out + (size_t)(first + t) * a.heads * VDIM + head * VDIM + lane * kEach;
            float o[kEach], sum_squares = 0.0f;
#pragma unroll
            for (int j = 0; j < kEach; ++j) {
                o[j] = o_s[t * VDIM + lane * kEach + j];
                sum_squares += o[j] * o[j];
            }
            const float inverse = rsqrtf(warp_sum(sum_squares) / (float)VDIM + a.eps);
#pragma unroll
            for (int j = 0; j < kEach; j += 2) {
                const float2 g = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&g_raw[u][j / 2]));
                const float y0 = o[j] * inverse * weights[j] * (g.x / (1.0f + expf(-g.x)));
                const float y1 = o[j + 1] * inverse * weights[j + 1] * (g.y / (1.0f + expf(-g.y)));
                *reinterpret_cast<__nv_bfloat162*>(dst + j) = __floats2bfloat162_rn(y0, y1);
            }
        }
    }
    if (MODE == GLA_LOCAL || last_segment) {
        float* target = MODE == GLA_LOCAL ? segment_state : state;
#pragma unroll
        for (int pair = 0; pair < 4; ++pair) {
            float* to = target + (size_t)row_of(pair) * VDIM + column0;
#pragma unroll
            for (int c = 0; c < 8; c += 4) {
                float4 low, high;
                tc5::halves_of(S[pair][c], low.x, high.x);
                tc5::halves_of(S[pair][c + 1], low.y, high.y);
                tc5::halves_of(S[pair][c + 2], low.z, high.z);
                tc5::halves_of(S[pair][c + 3], low.w, high.w);
                *reinterpret_cast<float4*>(to + c) = low;
                *reinterpret_cast<float4*>(to + VDIM + c) = high;
            }
            if (MODE == GLA_LOCAL && warp == 0 && lane < 8) {
                float low, high;
                tc5::halves_of(decay[pair], low, high);
                a.segment_decay[segment_index * kTileDim + row_of(pair)] = low;
                a.segment_decay[segment_index * kTileDim + row_of(pair) + 1] = high;
            }
        }
    }
}

// One token per sequence (decode): the state goes through the SM once, read and written 16 bytes at a time, and nothing else counts.
// Four warps share the 64 rows; a warp's load is a whole row of 128 columns (two rows of 64).  All of a thread's rows, the token's
// q, k, z, v and g are asked for before the first is used; with `settled` (the state was left by an earlier step, behind the copy of
// the batch that this step began with) the state is asked for while the kernel in front still runs.  64 sequences of 32 heads of 64 / 128
// (134 MB, 21 us of copying): a replayed step is 47.6 us longer with the tiled kernel, 18.0 with this one.
template <typename W, int VDIM>
__global__ void __launch_bounds__(128) gla_single_kernel(GlaArgs a, int settled) {
    pdl_trigger();
    if (!settled) pdl_wait();
    typedef __nv_bfloat16 T;
    constexpr int kLanes = VDIM / 4, kRowsAtOnce = 128 / kLanes, kRows = kTileDim / kRowsAtOnce;      // rows per thread
    __shared__ float q_s[kTileDim], k_s[kTileDim], alpha_s[kTileDim];
    __shared__ float4 part_s[4][kLanes];
    const int seq = blockIdx.x, head = blockIdx.y, token = a.q_start[seq];
    if (a.q_start[seq + 1] - token != 1) {
        if (settled) pdl_wait();
        return;
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int column = 4 * (threadIdx.x % kLanes), first_row = threadIdx.x / kLanes;
    float* state = a.state + ((size_t)a.state_slots[seq] * a.heads + head) * kTileDim * VDIM + (size_t)first_row * VDIM + column;
    float4 S[kRows];
#pragma unroll
    for (int r = 0; r < kRows; ++r) S[r] = *reinterpret_cast<const float4*>(state + (size_t)r * kRowsAtOnce * VDIM);
    if (settled) pdl_wait();
    const T* row = (const T*)a.proj + (size_t)token * a.row_width;
    float v[4], g[VDIM / 32] = {};
#pragma unroll
    for (int c = 0; c < 4; ++c) v[c] = Num<T>::load(row + a.v_offset + head * VDIM + column + c);
    if (warp == 0) {
#pragma unroll
        for (int j = 0; j < VDIM / 32; ++j) g[j] = Num<T>::load(row + a.g_offset + head * VDIM + lane * (VDIM / 32) + j);
    }
    if (threadIdx.x < kTileDim) {
        const int i = threadIdx.x;
        q_s[i] = Num<T>::load(row + a.q_offset + head * kTileDim + i) * a.q_scale;
        k_s[i] = Num<T>::load(row + a.k_offset + head * kTileDim + i);
        float zz = a.z[((size_t)token * a.heads + head) * kTileDim + i];
        if (a.z_bias) zz += a.z_bias[head * kTileDim + i];
        const float log_sigmoid = zz >= 0.0f ? -log1pf(expf(-zz)) : zz - log1pf(expf(zz));
        alpha_s[i] = expf(log_sigmoid * a.inverse_tau);
    }
    __syncthreads();
    float4 o = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
        const int i = first_row + r * kRowsAtOnce;
        const float alpha = alpha_s[i], k = k_s[i], q = q_s[i];
        S[r].x = fmaf(alpha, S[r].x, k * v[0]);
        S[r].y = fmaf(alpha, S[r].y, k * v[1]);
        S[r].z = fmaf(alpha, S[r].z, k * v[2]);
        S[r].w = fmaf(alpha, S[r].w, k * v[3]);
        *reinterpret_cast<float4*>(state + (size_t)r * kRowsAtOnce * VDIM) = S[r];
        o.x = fmaf(S[r].x, q, o.x);
        o.y = fmaf(S[r].y, q, o.y);
        o.z = fmaf(S[r].z, q, o.z);
        o.w = fmaf(S[r].w, q, o.w);
    }
    if (kLanes == 16) {      // two rows per warp
        o.x += __shfl_xor_sync(0xffffffffu, o.x, 16);
        o.y += __shfl_xor_sync(0xffffffffu, o.y, 16);
        o.z += __shfl_xor_sync(0xffffffffu, o.z, 16);
        o.w += __shfl_xor_sync(0xffffffffu, o.w, 16);
    }
    if (lane < kLanes) part_s[warp][lane] = o;
    __syncthreads();
    if (warp > 0) return;
    constexpr int kEach = VDIM / 32;
    const float* parts = reinterpret_cast<const float*>(part_s);
    float total[kEach], sum_squares = 0.0f;
#pragma unroll
    for (int j = 0; j < kEach; ++j) {
        const int at = lane * kEach + j;
        total[j] = ((parts[at] + parts[VDIM + at]) + parts[2 * VDIM + at]) + parts[3 * VDIM + at];
        sum_squares += total[j] * total[j];
    }
    const float inverse = rsqrtf(warp_sum(sum_squares) / (float)VDIM + a.eps);
    T* dst = (T*)a.out + ((size_t)token * a.heads + head) * VDIM + lane * kEach;
#pragma unroll
    for (int j = 0; j < kEach; ++j) {
        const float gate = g[j] / (1.0f + expf(-g[j]));
        Num<T>::store(dst + j, total[j] * inverse * Num<W>::load((const W*)a.weight + lane * kEach + j) * gate);
    }
}

// The scan between the passes: per (sequence, head), S_in(0) is the slot's state and S_in(k + 1) = D_k S_in(k) + S_local(k);
// S_in(k) takes S_local(k)'s place in the scratch.  One thread per cell of S: the cells are independent, and the
// segments' values are loaded a few ahead of the chain of multiply-adds that needs them.
__global__ void gla_scan_kernel(GlaArgs a) {
    pdl_trigger();
    pdl_wait();
    const int seq = blockIdx.x, head = blockIdx.y;
    const int tokens = a.q_start[seq + 1] - a.q_start[seq];
    if (tokens <= 0) return;
    const int segments = (tokens + a.segment - 1) / a.segment;
    const int cells = a.dim * a.vdim;
    const int cell = blockIdx.z * blockDim.x + threadIdx.x;
    if (cell >= cells) return;
    const int row = cell / a.vdim;
    float S = a.state[((size_t)a.state_slots[seq] * a.heads + head) * cells + cell];
    const size_t first = ((size_t)seq * a.max_segments) * a.heads + head;
    const size_t stride = a.heads;      // from one segment's index to the next's
    constexpr int AHEAD = 4;
    for (int k0 = 0; k0 < segments; k0 += AHEAD) {
        float local[AHEAD], decay[AHEAD];
#pragma unroll
        for (int u = 0; u < AHEAD; ++u) {
            const int k = k0 + u;
            const bool more = k + 1 < segments;
            const size_t index = first + (size_t)k * stride;
            local[u] = more ? a.segment_state[index * cells + cell] : 0.0f;
            decay[u] = more ? a.segment_decay[index * a.dim + row] : 0.0f;
        }
#pragma unroll
        for (int u = 0; u < AHEAD; ++u) {
            const int k = k0 + u;
            if (k < segments) {
                a.segment_state[(first + (size_t)k * stride) * cells + cell] = S;
                if (k + 1 < segments) S = fmaf(decay[u], S, local[u]);
            }
        }
    }
}

// Rows of S per thread: the smallest of 16, 32, 64, 128 with which the partitions that cover `dim` fit a block.
static int gla_rows_per_thread(int dim, int column_threads) {
    const int choices[4] = {16, 32, 64, 128};
    for (int c = 0; c < 4; ++c) {
        const int partitions = (dim + choices[c] - 1) / choices[c];
        // 128 rows of state per thread leave room for 256 threads' registers only
        if (partitions * column_threads <= (choices[c] == 128 ? 256 : 512)) return choices[c];
    }
    if ((dim + 127) / 128 * column_threads <= 512) return 129;      // 128 rows with 512 threads: the state spills
    return 0;
}

LLM_EXPORT int llm_gla_supports(int dim, int vdim) {
    if (dim <= 0 || vdim <= 0 || vdim > 512) return 0;
    return gla_rows_per_thread(dim, (vdim + 31) / 32 * 32) != 0;
}

// bfloat16 steps of heads with 64 key channels and 64 or 128 value channels: the tiled kernel, or the one for single tokens.
template <typename W, int VDIM>
int gla_tiles_launch(const GlaArgs& a, int n_seqs, bool segmented, int singles, int settled, cudaStream_t stream) {
    if (singles && !segmented) {
        llm_launch(gla_single_kernel<W, VDIM>, dim3(n_seqs, a.heads), 128, 0, stream, a, settled);
        return llm_check_launch("gla_recurrent");
    }
    const size_t shared = ((size_t)3 * GLA_TOKENS * kTileDim + (size_t)2 * GLA_TOKENS * VDIM) * sizeof(float);
    const dim3 grid(n_seqs, a.heads, segmented ? a.max_segments : 1);
    if (!segmented) {
        llm_launch(gla_tiles_kernel<W, VDIM, GLA_ONE_PASS>, grid, VDIM, shared, stream, a);
    } else {
        llm_launch(gla_tiles_kernel<W, VDIM, GLA_LOCAL>, grid, VDIM, shared, stream, a);
        llm_launch(gla_scan_kernel, dim3(n_seqs, a.heads, (a.dim * a.vdim + 255) / 256), 256, 0, stream, a);
        llm_launch(gla_tiles_kernel<W, VDIM, GLA_OUTPUT>, grid, VDIM, shared, stream, a);
    }
    return llm_check_launch("gla_recurrent");
}

// singles: every sequence of the step has one token (or none).  settled: the states were left by earlier steps, behind which the
// kernel launched just before this one was queued: they may be read without waiting for it.
LLM_EXPORT int llm_gla_recurrent(const void* proj, int row_width, int q_offset, int k_offset, int v_offset, int g_offset,
                                 const float* z, const float* z_bias, const void* weight, float* state, const int* state_slots,
                                 const int* q_start, void* out, int n_seqs, int heads, int dim, int vdim, float inverse_tau,
                                 float q_scale, float eps, int dtype, int weight_dtype, int segment, int max_segments,
                                 float* segment_state, float* segment_decay, int singles, int settled, cudaStream_t stream) {
    if (n_seqs == 0) return LLM_OK;
    if (!llm_gla_supports(dim, vdim) || heads <= 0) {
        llm_set_error("gla_recurrent: %d heads of %d key and %d value channels are not supported", heads, dim, vdim);
        return LLM_REFUSED;
    }
    GlaArgs a;
    a.proj = proj; a.row_width = row_width; a.q_offset = q_offset; a.k_offset = k_offset; a.v_offset = v_offset; a.g_offset = g_offset;
    a.z = z; a.z_bias = z_bias; a.weight = weight; a.state = state; a.state_slots = state_slots; a.q_start = q_start; a.out = out;
    a.heads = heads; a.dim = dim; a.vdim = vdim;
    a.column_threads = (vdim + 31) / 32 * 32;
    const int choice = gla_rows_per_thread(dim, a.column_threads);
    const int rows = choice == 129 ? 128 : choice;
    a.partitions = (dim + rows - 1) / rows;
    a.padded_dim = a.partitions * rows;
    a.inverse_tau = inverse_tau; a.q_scale = q_scale; a.eps = eps;
    a.segment = segment; a.max_segments = max_segments; a.segment_state = segment_state; a.segment_decay = segment_decay;
    const bool segmented = segment > 0;
    if (segmented && (max_segments <= 0 || !segment_state || !segment_decay)) {
        llm_set_error("gla_recurrent: the segmented form needs its scratch");
        return LLM_REFUSED;
    }
    // the tiled kernel reads rows and states in 16-byte pieces
    const bool pieces = aligned16(proj) && row_width % 8 == 0 && q_offset % 8 == 0 && k_offset % 8 == 0 && v_offset % 8 == 0 && g_offset % 8 == 0 && aligned16(z) && aligned16(out) &&
                        aligned16(state) && (!segmented || (aligned16(segment_state) && aligned16(segment_decay)));
    if (dtype == LLM_BF16 && (weight_dtype == LLM_F32 || weight_dtype == LLM_BF16) && dim == kTileDim && (vdim == 64 || vdim == 128) && pieces) {
        if (vdim == 64) return weight_dtype == LLM_F32 ? gla_tiles_launch<float, 64>(a, n_seqs, segmented, singles, settled, stream) : gla_tiles_launch<__nv_bfloat16, 64>(a, n_seqs, segmented, singles, settled, stream);
        return weight_dtype == LLM_F32 ? gla_tiles_launch<float, 128>(a, n_seqs, segmented, singles, settled, stream) : gla_tiles_launch<__nv_bfloat16, 128>(a, n_seqs, segmented, singles, settled, stream);
    }
    const int threads = a.partitions * a.column_threads;
    const size_t shared = ((size_t)3 * GLA_TOKENS * a.padded_dim + (size_t)GLA_TOKENS * vdim + (size_t)a.partitions * GLA_TOKENS * vdim) * sizeof(float);
    dim3 grid(n_seqs, heads, segmented ? max_segments : 1);
#define GLA_LAUNCH_MODE(R, MODE)                                                                                        \
    do {                                                                                                                \
        if (shared > 40 * 1024) {                                                                                       \
            const int status = llm_raise_shared_limit((const void*)gla_recurrent_kernel<T, W, R, MODE>, shared, "gla_recurrent"); \
            if (status != LLM_OK) return status;                                                                        \
        }                                                                                                               \
        llm_launch(gla_recurrent_kernel<T, W, R, MODE>, grid, threads, shared, stream, a);                              \
    } while (0)
#define GLA_LAUNCH(R)                                                                                                   \
    do {                                                                                                                \
        if (!segmented) {                                                                                               \
            GLA_LAUNCH_MODE(R, GLA_ONE_PASS);                                                                           \
        } else {                                                                                                        \
            GLA_LAUNCH_MODE(R, GLA_LOCAL);                                                                              \
            llm_launch(gla_scan_kernel, dim3(n_seqs, heads, (dim * vdim + 255) / 256), 256, 0, stream, a);                            \
            GLA_LAUNCH_MODE(R, GLA_OUTPUT);                                                                             \
        }                                                                                                               \
    } while (0)
    LLM_DISPATCH_DTYPE_WEIGHT(dtype, weight_dtype, {
        if (choice == 16) GLA_LAUNCH(16);
        else if (choice == 32) GLA_LAUNCH(32);
        else if (choice == 64) GLA_LAUNCH(64);
        else if (choice == 128) GLA_LAUNCH(128);
        else GLA_LAUNCH(129);
    });
#undef GLA_LAUNCH
#undef GLA_LAUNCH_MODE
    return llm_check_launch("gla_recurrent");
}
