// Launches of the kernels on pairs of SMs, for the dispatch of their single-CTA counterparts.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

namespace lb {

// attn_pair_sm100.cu. tq, tk, tv: the maps of attn_prefill_sm100.cu (boxes of 64 columns, 128 query rows or one page).
// -1: not for these sizes.
int pair_attn_launch(const CUtensorMap* tq, const CUtensorMap* tk, const CUtensorMap* tv, const int* cu_q, const int* ctx_lens,
                     const int* block_table, int table_width, int page, int n_seqs, int max_q_len, int Hq, int Hkv, int dk,
                     int dv, float scale_log2, void* out, int* status, cudaStream_t s);

}  // namespace lb
