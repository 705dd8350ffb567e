// Host launchers of the small element-wise operators that sit either side of every quantized linear in
// a decoder layer (residual add + RMSNorm, rotary embedding, SwiGLU).
#pragma once
#include <cuda_runtime.h>

namespace b2 {
int rmsnorm_launch(void* x, const void* r, const void* w, void* y, int T, int H, float eps, cudaStream_t s);
int rope_launch(void* q, void* k, const void* inv_freq, int T, int Hq, int Hk, int D, int pos0,
                long long q_stride, long long k_stride, cudaStream_t s);
int swiglu_launch(const void* gate, const void* up, void* out, int T, int I, cudaStream_t s);
int qkv_prefill_launch(void* qkv, const void* bias, const void* inv_freq, void* cache_k, void* cache_v, int T, int Hq,
                       int Hk, int D, int max_len, cudaStream_t s);
int swiglu_blocks_launch(const void* gu, void* out, int T, int I, int block, cudaStream_t s);
}  // namespace b2
