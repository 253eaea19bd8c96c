// What the general attention kernel (attention_generic.cu) and the 32-bit one (attention_f32.cu) are told of a step.
#pragma once

#include "common.cuh"

struct AttentionArgs {
    const void* q;        // [rows, ldq], head h at h*head_dim
    long long ldq;
    const void* k_step;   // keys of this step's rows [rows, ldkv], kv head g at g*head_dim; null: read the cache only
    const void* v_step;
    long long ldkv;
    const void* k_cache;  // storage of this schedule entry (may be null when every key is in the step)
    const void* v_cache;
    CacheGeometry cache;
    void* out;            // [rows, ldo]
    long long ldo;
    const int* row_seq;   // [rows] (-1: padding row: output zeros)
    const int* row_pos;
    const int* seq_slot;
    const int* seq_start; // tokens in the cache before this step
    const int* seq_row0;  // first packed row of the sequence
    int rows, heads, kv_heads, head_dim, window;  // window 0: every earlier key is visible
    float scale;
    float softcap;        // > 0: a score s becomes softcap * tanh(s / softcap)
    const float* slopes;  // [heads] or null: head h adds slopes[h] * (key position - query position) to a score
    int value_dim;        // width of a value head and of a head of `out` (0: head_dim), at most 256
    const float* sinks;   // [heads] or null: exp(sinks[h]) is added to head h's softmax denominator (a key that
                          // every row sees, with that score as it is, unscaled, and no value)
    const void* gate;     // [rows, ldg] or null: head h of a row is multiplied by sigmoid(gate[row, h])
    long long ldg;
    const float* weight_bias;  // [heads] or null: the weight of a key is sigmoid(score + weight_bias[h]) instead of its
                               // share of a softmax (nothing is normalised over the keys)
    int chunk;                 // > 0: only keys of the query's own run of `chunk` positions are seen
    float out_scale;           // the result is multiplied by it
    int tied;                  // k_step / k_cache hold keys before their norm, which are the values too (v_step, v_cache name
                               // the same rows); a score takes the factor 1 / sqrt(mean square of the key + key_eps)
    float key_eps;
    const float* distance_bias;   // [heads, bias_stride] or null: entry min(p - u, bias_last) of head h's row is added to a score
    int bias_stride, bias_last;
    const void* element_gate;     // [rows, ld_element_gate] or null: the result is multiplied by sigmoid of it, element by element
    long long ld_element_gate;
};
