// GEMM launches that do not fill the chip (gemm_split.cu): called by lb_gemm_grouped_epi, and by tests that name the form.
#pragma once
#include "common.cuh"

extern "C" int lb_gemm_split(int n, const void* const* A, const void* const* B, void* const* C, const int* M, const int* N, const int* K,
                             const long long* lda, const long long* ldb, const long long* ldc, const int* a_mn, const int* b_mn,
                             const int* accumulate, const int* epi, void* const* C2, const long long* ldc2, const int* half, int ks, void* stream);
int gemm_split_parts(int n, const int* M, const int* N, const int* K, int sms, long long list_time);
