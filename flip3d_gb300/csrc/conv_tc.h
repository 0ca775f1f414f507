/*
 * conv_tc.h — the U-Net's forward 3x3x3 convolution on the tcgen05 tensor
 * cores (k_conv_tc.cu). Activations are BF16 [sample][cell][channel] with
 * cells x-major; weights come in the layout of conv_tc_weight.
 */
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>

/* whether conv_tc_launch handles this level size and channel counts */
bool conv_tc_supported(int n, int cin, int cout);

/* Where weight e of W[tap][ci][co] (tap = (di*3 + dj)*3 + dk) lies among the 27*cin*cout
 * BF16 of conv_tc_launch's operand: per stage (di, chunk c) and tap t9 = dj*3 + dk a
 * block of cout*32 bytes: two K-halves of cout/8 core matrices (8 output
 * channels x 8 input channels, 16-byte rows). */
__device__ __forceinline__ int conv_tc_weight(int cin, int cout, int e) {
  const int co = e % cout, ci = (e / cout) % cin, tap = e / (cout * cin);
  const int di = tap / 9, t9 = tap % 9;
  const int c = ci / 16, kk = ci % 16, h = kk / 8, col = kk % 8, g = co / 8, r = co % 8;
  return (((di * (cin / 16) + c) * 9 + t9) * cout * 32 + (h * (cout / 8) + g) * 128 + r * 16) / 2 +
         col;
}

/* Y = (relu)(conv3x3x3(X, W) + bias) over batch samples of an n^3 grid
 * (bias may be null). An expired bounded wait inside the kernel sets *err
 * to 1; the launch itself reports configuration errors. */
cudaError_t conv_tc_launch(cudaStream_t st, int n, int batch, int cin, int cout,
                           const __nv_bfloat16 *X, const __nv_bfloat16 *Wtc, const float *bias,
                           __nv_bfloat16 *Y, int relu, int *err);

/* one-time per-device setup (shared-memory limits); 0 on success */
int conv_tc_init_device();
