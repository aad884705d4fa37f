// The form of bias + norm + rotation + cache write that moves 16-byte pieces (norm_rope_units.cu), for the launchers that use it.
#pragma once
#include "common.cuh"

struct UnitPieces {
    __nv_bfloat16* qkv;             // [tokens, row_width]: [units of queries | units of keys | values | ...]
    int row_width;
    const float* bias;              // of the columns used, or null
    const void *q_weight, *k_weight;    // norm weights of a unit, or null
    int weight_is_f32;
    float eps;
    const float* inv_freq;          // [dim / 2], or null: whole units turn, halves paired, or nothing does
    float magnitude;                // on cos and sin
    const int *positions, *seq_of_token, *block_tables;
    int max_blocks;
    __nv_bfloat16 *k_pages, *v_pages;
    int n_kv_heads, maps;           // a key head is `maps` units
    int q_cols, dim, value_dim;     // columns of queries; elements of a query or key unit (64 or 128); of a value head
    int page_size, num_pages, write_cache;
    int* error_flag;
};

// Whether the sizes and alignments are ones the form takes.
bool unit_pieces_take(const UnitPieces& p);
int unit_pieces_launch(const UnitPieces& p, int n_tokens, cudaStream_t stream);
