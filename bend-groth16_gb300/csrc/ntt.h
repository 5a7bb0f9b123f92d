// NTT / QAP interface (see ntt.cu)
#pragma once
#include "common.cuh"

namespace bg {

NttTables& ntt_tables(Ctx& ctx, int L);
// device bytes of the tables of a 2^L domain
size_t ntt_table_bytes(int L);
// in-place transform of 2^L packed Fr, natural order in and out; mode = BG_NTT_*
void ntt_run(Ctx& ctx, cudaStream_t st, uint32_t* d_data, int L, int mode);
// h from evaluation vectors a, b, c (overwritten); d_h receives 2^L coefficients, Montgomery or
// canonical
void qap_h_run(Ctx& ctx, cudaStream_t st, uint32_t* d_a, uint32_t* d_b, uint32_t* d_c, uint32_t* d_h, int L,
               bool canonical);

}  // namespace bg
