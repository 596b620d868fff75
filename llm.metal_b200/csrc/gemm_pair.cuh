// The pair-of-SMs form of the 16-bit tensor-core products (gemm_pair.cu).
#pragma once
#include "../../include/llmb200_train_kernels.h"

#include <cuda_runtime.h>

struct PairShape { int bn, splits; };
// How pairs would take a product, and the modelled clocks (1e30: not at all, 128 rows or fewer, or fewer than 256 columns).
double gemm_pair_shape(int M, int N, int K, bool may_split, PairShape *out);
// Operands checked by the caller; fmt 0: binary16, 1: bfloat16.
int gemm_pair_launch(const b200_gemm_args *a, int fmt, const PairShape &sh, cudaStream_t st);
