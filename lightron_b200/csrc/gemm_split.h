// GEMM launches that do not fill the chip (gemm_split.cu): called by lb_gemm_grouped_epi, and by tests that name the form.
#pragma once
#include "common.cuh"

// Epilogue 4 (no entry point takes it but lb_gemm_rope): the first `cols` columns of C are heads of d columns whose pairs (2i, 2i + 1) are rotated
// as lb_rope does, from the values that a stored C would have; row r is token r of sequences of S tokens.
struct RopeArgs {
  const float *cos, *sin;
  const int* positions;      // [S] or null: the token's place in its sequence
  int S, d, cols;
};
__device__ __forceinline__ int rope_position(const RopeArgs& r, int row) {
  const int s = row % r.S;
  return r.positions ? r.positions[s] : s;
}
// Cosines and sines (4 and 4) of 8 columns of C, from `col` (a multiple of 8), of a row at that position: what rope_rotate8() takes
__device__ __forceinline__ void rope_load8(const RopeArgs& r, int pos, int col, float* cs) {
  const int at = pos * (r.d >> 1) + ((col % r.d) >> 1);
  *reinterpret_cast<float4*>(cs) = *reinterpret_cast<const float4*>(r.cos + at);
  *reinterpret_cast<float4*>(cs + 4) = *reinterpret_cast<const float4*>(r.sin + at);
}
extern "C" int lb_gemm_split(int n, const void* const* A, const void* const* B, void* const* C, const int* M, const int* N, const int* K,
                             const long long* lda, const long long* ldb, const long long* ldc, const int* a_mn, const int* b_mn,
                             const int* accumulate, const int* epi, void* const* C2, const long long* ldc2, const int* half, int ks, void* stream);
// The same with the rotation of epilogue 4 (n = 1), or with `rope` null.
int gemm_split_rope(int n, const void* const* A, const void* const* B, void* const* C, const int* M, const int* N, const int* K,
                    const long long* lda, const long long* ldb, const long long* ldc, const int* a_mn, const int* b_mn,
                    const int* accumulate, const int* epi, void* const* C2, const long long* ldc2, const int* half, int ks, const RopeArgs* rope,
                    void* stream);
int gemm_split_parts(int n, const int* M, const int* N, const int* K, bool activation, int sms, long long list_time, double* us);
