// The product on pairs of SMs (gemm_pair.cu), as the persistent product (gemm_tc.cu) calls it.
#pragma once
#include "common.cuh"

#define GEMM_STORE 0
#define GEMM_ACCUM 1
#define GEMM_SWIGLU 2
// More forms of the kernels, instantiations of their own so that the three above are what they were: the gated form
// with a ReLU gate, out = up * relu(gate), and the storing forms with out = relu(alpha * sum)^2 and out = xIELU(alpha * sum).
#define GEMM_REGLU 3
#define GEMM_STORE_RELU2 4
#define GEMM_STORE_XIELU 5
#define GEMM_GATED(MODE) ((MODE) == GEMM_SWIGLU || (MODE) == GEMM_REGLU)

// Expected time (us) of the product on pairs; out_bytes: of an output element.
double gemm_pair_estimate(int mode, int M, int N, int K, int out_bytes, int sm_count);

// `mode` is one of the forms above; out and ldo must be addressable by TMA (16-byte aligned); n_tile 0: chosen by the sizes.
int gemm_pair_launch(int mode, const void* X, int ldx, const void* W, int ldw, void* out, int out_dtype, int ldo, int M, int N,
                     int K, float alpha, int sm_count, int n_tile, float act_p, float act_n, int* error_flag, cudaStream_t stream);
