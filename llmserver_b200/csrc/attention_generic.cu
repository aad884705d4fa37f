// Attention over the paged cache, any sizes, 32-bit arithmetic: the kernel of the true 32-bit path
// and the fallback of the bfloat16 path for head sizes its tensor-core kernels refuse.
//
// A block of four warps per (query token, query head), or a warp where there are many.  The query at absolute position p sees keys
// max(0, p - window + 1) .. p of its own sequence (window 0 = all), read through the sequence's
// block table; the new tokens' keys are already in the cache when this runs.  Scores, the running
// maximum, the normaliser and the output accumulate in 32-bit with the online-softmax recurrence
// the reference's paged path uses (utils/attention.py:75-96, utils/paged_attention.py:60-75);
// query head h reads kv head h / group (utils/attention.py:186-190); scale multiplies the dot
// product (utils/architecture.py:105).
//
// Keys are visited 32 at a time from the first visible one, each lane owning one key's dot
// product; part w of four takes rounds w, w + 4, ... and the parts are merged in their order, whether four warps make them or one.
// So the order of every sum depends only on the query's position: the result for a token
// is bit-identical however the prompt was cut into steps and whatever else is in the batch.
//
// Values may have another size than keys (`value_dim`; the output then has Hq * value_dim columns).  With `sinks`
// (one 32-bit number per query head) the softmax's denominator also holds exp(sinks[h]): a score without a key
// and without a value, not scaled, counted once.
//
// With `chunk` > 0 the sequence is cut into chunks of that many positions and a query sees the keys of its own chunk
// only (from (p / chunk) * chunk on).  With `bias` (32-bit [Hq, bias_len]) the score of the key n positions back gets
// bias[h][min(n, bias_len - 1)] added, which the scale does not multiply.
//
// With `keep` > 0 a windowed query also sees the sequence's first `keep` positions, at their true distances; they are
// visited in front of the window's keys.  With `gate` the results are multiplied by sigmoid(gate[token * gate_stride + h *
// value_dim + d]), formed in 32-bit, before their one rounding.
#include "common.cuh"

#define ATTN_MAX_D 512

namespace {

// The dot product of a lane's key row with the query, one fused multiply-add per element in ascending order.  VECTOR: 16 bytes
// at a time, eight of them asked for before the first is used.
template <typename T, bool VECTOR>
__device__ __forceinline__ float row_dot(const float* q_row, const T* k_row, int head_dim) {
    float dot = 0.0f;
    if constexpr (VECTOR) {
        constexpr int kCount = Vec16<T>::kCount, kDeep = 8;
        int d = 0;
        for (; d + kDeep * kCount <= head_dim; d += kDeep * kCount) {
            uint4 raw[kDeep];
#pragma unroll
            for (int i = 0; i < kDeep; ++i) raw[i] = *reinterpret_cast<const uint4*>(k_row + d + i * kCount);
#pragma unroll
            for (int i = 0; i < kDeep; ++i) {
                float k[kCount];
                Vec16<T>::load(reinterpret_cast<const T*>(&raw[i]), k);
#pragma unroll
                for (int j = 0; j < kCount; ++j) dot = fmaf(q_row[d + i * kCount + j], k[j], dot);
            }
        }
        for (; d < head_dim; d += kCount) {
            float k[kCount];
            Vec16<T>::load(k_row + d, k);
#pragma unroll
            for (int j = 0; j < kCount; ++j) dot = fmaf(q_row[d + j], k[j], dot);
        }
    } else {
#pragma unroll 8
        for (int d = 0; d < head_dim; ++d) dot = fmaf(q_row[d], Num<T>::load(k_row + d), dot);
    }
    return dot;
}

}  // namespace

// COLUMNS: value elements per lane, the least power of two that covers the value size.  What bounds the kernel for few tokens is
// the chain of dependent loads per 32 keys (table entry, key row, value rows); so the value rows of a round are asked for,
// kAhead at a time, before the weights that multiply them are known, and the table entry of the next round with them.  With
// 150 keys, heads of 32 and 4 tokens a launch took 52 us when the loads were issued one by one and the accumulator had 16
// columns for every size, and added 11.3 us to a replayed step when one warp walked all five rounds; with the rounds dealt to four
// warps it adds 8.6.
//
// LONE: a warp makes all four parts of its (token, head), round after round, and keeps each part's sums.  Four warps per pair only help
// while the GPU has room for them and a pair has rounds for all: with many pairs they crowd each other out of the L1 cache (the more,
// the wider the values) and merge through shared memory for nothing, and at a prompt's first positions most have no round.  us a
// launch, four warps / one; 32-bit prompts of 6 heads of 32: 128 tokens 8.7 / 11.8, 683 95 / 105, 2048 722 / 703, 4096 2823 / 2594,
// 2048 behind a window of 64 keys 74 / 44; 16 heads of 64: 128 tokens 24 / 35, 512 222 / 232, 2048 3187 / 2961; 32 heads of 128: 32
// tokens 17.7 / 11.3, 32 behind 1000 278 / 372, 96 behind 1000 717 / 605, 512 879 / 773; 8 heads of 192: 2048 tokens 8096 / 4755;
// bfloat16, 32 heads of 96: 32 tokens behind 4000 688 / 1054, 64 1362 / 1283, 1024 2192 / 1448.  Held to six blocks an SM (with values
// of up to 128) the one-warp form is 2 to 20 % faster than left alone.
constexpr int kParts = 4;
constexpr int kManySums = 8192;       // pairs x columns from which a warp makes all parts
constexpr int kFewKeys = 64, kManyShortPairs = 2048;      // the same with no more than two rounds: from so many pairs; with one: always
// Two parts' sums, each times what the common maximum makes of its own.
__device__ __forceinline__ float merged(float a, float a_weight, float b, float b_weight) { return fmaf(a, a_weight, b * b_weight); }

template <typename T, int COLUMNS, bool VECTOR, bool LONE>
__global__ void __launch_bounds__(kParts * 32, !LONE ? 1 : COLUMNS <= 4 ? 6 : COLUMNS == 8 ? 4 : 3) attention_generic_kernel(const T* __restrict__ q, int q_stride, const T* __restrict__ k_pages,
                                         const T* __restrict__ v_pages, const int* __restrict__ block_tables,
                                         int max_blocks, const int* __restrict__ seq_of_token,
                                         const int* __restrict__ positions, T* __restrict__ out, int n_q_heads,
                                         int n_kv_heads, int head_dim, int value_dim, int page_size, int num_pages,
                                         float scale, int window, const float* __restrict__ sinks,
                                         int chunk, const float* __restrict__ bias, int bias_len, int keep,
                                         const T* __restrict__ gate, int gate_stride, int* __restrict__ error_flag) {
    constexpr int kAhead = COLUMNS >= 16 ? 2 : 32 / COLUMNS;      // value rows in flight: 32 registers per lane
    pdl_trigger();   // let the next kernel start launching
    // LONE: [4][head_dim]; else [head_dim], then what warps 1 .. 3 leave: [3][maximum, normaliser, 32 * COLUMNS sums]
    extern __shared__ float q_shared[];
    const int token = blockIdx.x;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int head = LONE ? blockIdx.y * kParts + warp : blockIdx.y;
    if (LONE && head >= n_q_heads) return;
    const int kv_head = head / (n_q_heads / n_kv_heads);
    // A step's positions and block tables come from the host, or from a kernel that does not let its successors start early: they
    // are complete when this kernel starts, and are asked for while the kernel in front still runs.
    const int position = positions[token];
    const int* table = block_tables + (size_t)seq_of_token[token] * max_blocks;

    float* q_row = q_shared + (LONE ? warp * head_dim : 0);

    // of the parts that this warp makes; the part whose round comes next is in front
    constexpr int kHeld = LONE ? kParts : 1;
    float accumulators[kHeld][COLUMNS], maxima[kHeld], normalisers[kHeld];
#pragma unroll
    for (int h = 0; h < kHeld; ++h) {
        maxima[h] = -INFINITY, normalisers[h] = 0.0f;
#pragma unroll
        for (int i = 0; i < COLUMNS; ++i) accumulators[h][i] = 0.0f;
    }
    float (&accumulator)[COLUMNS] = accumulators[0];
    float &running_max = maxima[0], &normaliser = normalisers[0];
    auto next_part = [&] {
        if constexpr (LONE) {
            const float front_max = maxima[0], front_normaliser = normalisers[0];
#pragma unroll
            for (int h = 0; h + 1 < kHeld; ++h) maxima[h] = maxima[h + 1], normalisers[h] = normalisers[h + 1];
            maxima[kHeld - 1] = front_max, normalisers[kHeld - 1] = front_normaliser;
#pragma unroll
            for (int i = 0; i < COLUMNS; ++i) {
                const float front = accumulators[0][i];
#pragma unroll
                for (int h = 0; h + 1 < kHeld; ++h) accumulators[h][i] = accumulators[h + 1][i];
                accumulators[kHeld - 1][i] = front;
            }
        }
    };

    int first = (window > 0 && position - window + 1 > 0) ? position - window + 1 : 0;
    if (chunk > 0) first = max(first, position / chunk * chunk);
    const int kept = min(keep, first);      // keys 0 .. kept - 1, then first .. position
    const int count = kept + position - first + 1;
    auto key_of = [&](int index) { return index < kept ? index : first + index - kept; };
    constexpr int kStride = LONE ? 32 : 32 * kParts;
    const int first_base = LONE ? 0 : 32 * warp;
    int next_page = first_base + lane < count ? table[key_of(first_base + lane) / page_size] : 0;
    pdl_wait();      // everything before this kernel in the stream is complete and visible
    const T* q_src = q + (size_t)token * q_stride + (size_t)head * head_dim;
    for (int i = LONE ? lane : threadIdx.x; i < head_dim; i += kStride) q_row[i] = Num<T>::load(q_src + i);
    if (LONE) __syncwarp();      // the query's row
    else __syncthreads();
    for (int base = first_base; base < count; base += kStride) {
        const int index = base + lane;
        const int key = key_of(index);
        const bool valid = index < count;
        int page = next_page;
        if (index + kStride < count) next_page = table[key_of(index + kStride) / page_size];
        if (valid && (unsigned)page >= (unsigned)num_pages) {      // no page of the pool: report it, read page 0 instead
            if (error_flag) atomicExch(error_flag, 5);
            page = 0;
        }
        // this lane's key's slot in the pages: its key row lies at offset * head_dim, its value row at offset * value_dim
        const long long offset = valid ? ((long long)page * n_kv_heads + kv_head) * page_size + key % page_size : 0;
        const int in_chunk = min(32, count - base);
        float ahead[kAhead][COLUMNS];
        auto ask = [&](int j0) {      // value rows j0 .. j0 + kAhead - 1 of the round
#pragma unroll
            for (int j = 0; j < kAhead; ++j) {
                const long long row = __shfl_sync(0xffffffffu, offset, j0 + j);
                const T* v_row = v_pages + row * value_dim;
#pragma unroll
                for (int i = 0; i < COLUMNS; ++i) {
                    const int d = lane + 32 * i;
                    ahead[j][i] = j0 + j < in_chunk && d < value_dim ? Num<T>::load(v_row + d) : 0.0f;
                }
            }
        };
        ask(0);
        float score = -INFINITY;
        if (valid) {
            score = row_dot<T, VECTOR>(q_row, k_pages + offset * head_dim, head_dim) * scale;
            if (bias) score += bias[(size_t)head * bias_len + min(position - key, bias_len - 1)];
        }
        const float chunk_max = warp_max(score);
        const float new_max = fmaxf(running_max, chunk_max);
        // (a round may hold nothing but scores of -inf, which a bias can give: no weight, nothing to correct)
        const float correction = running_max == new_max ? 1.0f : expf(running_max - new_max);  // 0 on the first chunk
        const float weight = valid && score != -INFINITY ? expf(score - new_max) : 0.0f;
        normaliser = normaliser * correction + warp_sum(weight);
#pragma unroll
        for (int i = 0; i < COLUMNS; ++i) accumulator[i] *= correction;
        for (int j0 = 0; j0 < in_chunk; j0 += kAhead) {
            if (j0) ask(j0);
#pragma unroll
            for (int j = 0; j < kAhead; ++j) {
                const float w = __shfl_sync(0xffffffffu, weight, j0 + j);
                if (j0 + j < in_chunk) {
#pragma unroll
                    for (int i = 0; i < COLUMNS; ++i) accumulator[i] = fmaf(w, ahead[j][i], accumulator[i]);
                }
            }
        }
        running_max = new_max;
        next_part();
    }
    const int rounds = (count + 31) / 32;
    if constexpr (LONE) {
        for (int turn = rounds; turn % kParts != 0; ++turn) next_part();      // part 0 is in front again
#pragma unroll
        for (int other = 1; other < kParts; ++other) {
            if (other >= rounds || (maxima[other] == -INFINITY && normalisers[other] == 0.0f)) continue;
            const float new_max = fmaxf(running_max, maxima[other]);
            const float correction = running_max == new_max ? 1.0f : expf(running_max - new_max);
            const float weight = maxima[other] == new_max ? 1.0f : expf(maxima[other] - new_max);
            normaliser = merged(normaliser, correction, normalisers[other], weight);
#pragma unroll
            for (int i = 0; i < COLUMNS; ++i) accumulator[i] = merged(accumulator[i], correction, accumulators[other][i], weight);
            running_max = new_max;
        }
    } else if (rounds > 1) {      // warps 1 .. 3 leave what they have; warp 0 adds it in their order
        float* parts = q_shared + head_dim;
        constexpr int kPart = 2 + 32 * COLUMNS;
        if (warp > 0) {
            float* part = parts + (warp - 1) * kPart;
            if (lane == 0) {
                part[0] = running_max;
                part[1] = normaliser;
            }
#pragma unroll
            for (int i = 0; i < COLUMNS; ++i) part[2 + lane + 32 * i] = accumulator[i];
        }
        __syncthreads();
        if (warp == 0) {
            for (int other = 1; other < kParts && other < rounds; ++other) {
                const float* part = parts + (other - 1) * kPart;
                if (part[0] == -INFINITY && part[1] == 0.0f) continue;
                const float new_max = fmaxf(running_max, part[0]);
                const float correction = running_max == new_max ? 1.0f : expf(running_max - new_max);
                const float weight = part[0] == new_max ? 1.0f : expf(part[0] - new_max);
                normaliser = merged(normaliser, correction, part[1], weight);
#pragma unroll
                for (int i = 0; i < COLUMNS; ++i) accumulator[i] = merged(accumulator[i], correction, part[2 + lane + 32 * i], weight);
                running_max = new_max;
            }
        }
    }
    if (!LONE && warp > 0) return;
    if (sinks) {      // one more term of the denominator; it has no value, so the sums only shrink
        const float sink = sinks[head];
        const float new_max = fmaxf(running_max, sink);
        const float correction = expf(running_max - new_max);
        normaliser = normaliser * correction + expf(sink - new_max);
#pragma unroll
        for (int i = 0; i < COLUMNS; ++i) accumulator[i] *= correction;
    }
    T* dst = out + (size_t)token * n_q_heads * value_dim + (size_t)head * value_dim;
    const float inverse = 1.0f / normaliser;
#pragma unroll
    for (int i = 0; i < COLUMNS; ++i) {
        const int d = lane + 32 * i;
        if (d < value_dim) {
            float value = accumulator[i] * inverse;
            if (gate) value /= 1.0f + expf(-Num<T>::load(gate + (size_t)token * gate_stride + (size_t)head * value_dim + d));
            Num<T>::store(dst + d, value);
        }
    }
}

// max_keys: no token has more keys than this (0: not known); it only decides between forms that give the same bits.
LLM_EXPORT int llm_attention_generic(const void* q, int q_stride, const void* k_pages, const void* v_pages,
                                     const int* block_tables, int max_blocks, const int* seq_of_token,
                                     const int* positions, void* out, int n_tokens, int n_q_heads, int n_kv_heads,
                                     int head_dim, int value_dim, int page_size, int num_pages, float scale, int window,
                                     const float* sinks, int chunk, const float* bias, int bias_len, int keep, const void* gate, int gate_stride,
                                     int max_keys, int* error_flag, int dtype, cudaStream_t stream) {
    if (n_tokens == 0) return LLM_OK;
    if (head_dim > ATTN_MAX_D || head_dim <= 0) {
        llm_set_error("attention_generic: head_dim %d is outside 1..%d", head_dim, ATTN_MAX_D);
        return LLM_REFUSED;
    }
    if (value_dim > ATTN_MAX_D || value_dim <= 0) {
        llm_set_error("attention_generic: the value size %d is outside 1..%d", value_dim, ATTN_MAX_D);
        return LLM_REFUSED;
    }
    if (num_pages <= 0) {
        llm_set_error("attention_generic: the page pool has %d pages", num_pages);
        return LLM_REFUSED;
    }
    if (n_kv_heads <= 0 || n_q_heads % n_kv_heads) {
        llm_set_error("attention_generic: %d query heads are no multiple of %d kv heads", n_q_heads, n_kv_heads);
        return LLM_REFUSED;
    }
    if (chunk < 0 || (bias && bias_len <= 0) || keep < 0 || (keep > 0 && chunk > 0)) {
        llm_set_error("attention_generic: a chunk of %d positions, a bias of %d distances or %d kept positions", chunk, bias_len, keep);
        return LLM_REFUSED;
    }
    if (n_q_heads > kParts * 65535) {
        llm_set_error("attention_generic: %d query heads are too many for one launch", n_q_heads);
        return LLM_REFUSED;
    }
    const int columns = value_dim <= 32 ? 1 : value_dim <= 64 ? 2 : value_dim <= 128 ? 4 : value_dim <= 256 ? 8 : 16;
    long long keys = max_keys > 0 ? max_keys : 1LL << 40;
    if (window > 0) keys = min(keys, (long long)window + keep);
    if (chunk > 0) keys = min(keys, (long long)chunk);
    const long long pairs = (long long)n_tokens * n_q_heads;
    const bool lone = pairs * columns >= kManySums || keys <= 32 || (keys <= kFewKeys && pairs >= kManyShortPairs) || n_q_heads > 65535;
    const dim3 grid(n_tokens, lone ? (n_q_heads + kParts - 1) / kParts : n_q_heads);
    const size_t shared = (lone ? (size_t)kParts * head_dim : (size_t)head_dim + (kParts - 1) * (2 + 32 * columns)) * sizeof(float);
    // key rows in 16-byte pieces where every row starts on such a boundary
    const int count = dtype == LLM_F32 ? 4 : 8;
    const bool vector = head_dim % count == 0 && aligned16(k_pages);
#define LLM_GENERIC(COLUMNS)                                                                                                       \
    LLM_DISPATCH_DTYPE(dtype, llm_launch(lone ? (vector ? attention_generic_kernel<T, COLUMNS, true, true> : attention_generic_kernel<T, COLUMNS, false, true>) : \
                                                vector ? attention_generic_kernel<T, COLUMNS, true, false> : attention_generic_kernel<T, COLUMNS, false, false>, \
                                         grid, kParts * 32, shared, stream, (const T*)q, q_stride, (const T*)k_pages, (const T*)v_pages,     \
                                         block_tables, max_blocks, seq_of_token, positions, (T*)out, n_q_heads, n_kv_heads, head_dim,       \
                                         value_dim, page_size, num_pages, scale, window, sinks, chunk, bias, bias_len, keep,                \
                                         (const T*)gate, gate_stride, error_flag))
    if (columns == 1) LLM_GENERIC(1);
    else if (columns == 2) LLM_GENERIC(2);
    else if (columns == 4) LLM_GENERIC(4);
    else if (columns == 8) LLM_GENERIC(8);
    else LLM_GENERIC(16);
#undef LLM_GENERIC
    return llm_check_launch("attention_generic");
}
