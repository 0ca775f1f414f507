/*
 * Every plan (lines per unit, pipeline stages) that the tcgen05 convolution
 * offers for a shape, against a plain convolution. The values are small
 * integers: each sum is below 2^24, so FP32 holds it exactly in any order and
 * the BF16 outputs have to be equal bit for bit.
 *
 *   conv_lines_check n cin cout batch  ->  "plans <count> eight <count> bad <count>"
 * (eight: plans of eight lines).
 */
#include "k_conv_tc.cu"

#include <cstdlib>

__global__ void k_fill(size_t count, unsigned salt, bf16 *out, float *outf) {
  const size_t e = (size_t)blockIdx.x * 256 + threadIdx.x;
  if (e >= count) return;
  unsigned h = (unsigned)e * 2654435761u + salt;
  h ^= h >> 15;
  h *= 2246822519u;
  h ^= h >> 13;
  const float v = (float)((int)(h % 9u) - 4);
  if (out) out[e] = __float2bfloat16(v);
  if (outf) outf[e] = v;
}

__global__ void k_pack_check(int cin, int cout, const float *W, bf16 *out) {
  const int e = blockIdx.x * 256 + threadIdx.x;
  if (e < 27 * cin * cout) out[conv_tc_weight(cin, cout, e)] = __float2bfloat16(W[e]);
}

__global__ void k_plain(int n, int batch, int cin, int cout, const bf16 *X, const float *W,
                        const float *bias, bf16 *Y) {
  const size_t e = (size_t)blockIdx.x * 256 + threadIdx.x, n3 = (size_t)n * n * n;
  if (e >= n3 * batch * cout) return;
  const int co = (int)(e % cout);
  const size_t vc = e / cout, s = vc / n3, v = vc % n3;
  const int i = (int)(v / ((size_t)n * n)), j = (int)(v / n % n), k = (int)(v % n);
  float a = bias[co];
  for (int tap = 0; tap < 27; tap++) {
    const int x = i + tap / 9 - 1, y = j + tap / 3 % 3 - 1, z = k + tap % 3 - 1;
    if (x < 0 || x >= n || y < 0 || y >= n || z < 0 || z >= n) continue;
    const bf16 *row = X + (s * n3 + ((size_t)x * n + y) * n + z) * cin;
    for (int ci = 0; ci < cin; ci++)
      a += __bfloat162float(row[ci]) * W[((size_t)tap * cin + ci) * cout + co];
  }
  Y[e] = __float2bfloat16(fmaxf(a, 0.0f));
}

__global__ void k_differ(size_t count, const uint16_t *a, const uint16_t *b,
                         unsigned long long *bad) {
  const size_t e = (size_t)blockIdx.x * 256 + threadIdx.x;
  if (e < count && a[e] != b[e]) atomicAdd(bad, 1ull);
}

int main(int argc, char **argv) {
  if (argc < 5) return 2;
  const int n = atoi(argv[1]), cin = atoi(argv[2]), cout = atoi(argv[3]), batch = atoi(argv[4]);
  const size_t cells = (size_t)n * n * n * batch, nw = (size_t)27 * cin * cout;
  const auto grid = [](size_t c) { return (unsigned)((c + 255) / 256); };
  bf16 *X, *Wt, *Y, *R;
  float *W, *bias;
  int *err;
  unsigned long long *bad;
  if (cudaMalloc(&X, cells * cin * 2) || cudaMalloc(&Wt, nw * 2) || cudaMalloc(&Y, cells * cout * 2) ||
      cudaMalloc(&R, cells * cout * 2) || cudaMalloc(&W, nw * 4) || cudaMalloc(&bias, cout * 4) ||
      cudaMalloc(&err, 4) || cudaMalloc(&bad, 8))
    return 3;
  cudaMemset(err, 0, 4);
  cudaMemset(bad, 0, 8);
  k_fill<<<grid(cells * cin), 256>>>(cells * cin, 1u, X, nullptr);
  k_fill<<<grid(nw), 256>>>(nw, 77u, nullptr, W);
  k_fill<<<1, 256>>>((size_t)cout, 5u, nullptr, bias);
  k_pack_check<<<grid(nw), 256>>>(cin, cout, W, Wt);
  k_plain<<<grid(cells * cout), 256>>>(n, batch, cin, cout, X, W, bias, R);
  if (cudaDeviceSynchronize() != cudaSuccess) return 4;
  int plans = 0, eight = 0;
  for (const auto &c : tc_candidates(n, cin, cout, batch)) {
    cudaMemset(Y, 0xff, cells * cout * 2);
    if (tc_launch_one(0, n, batch, cin, cout, X, Wt, bias, Y, 1, err, c.first, c.second) !=
        cudaSuccess)
      return 5;
    k_differ<<<grid(cells * cout), 256>>>(cells * cout, (const uint16_t *)Y, (const uint16_t *)R,
                                          bad);
    plans++;
    eight += c.first == 8;
  }
  int e = 0;
  unsigned long long b = 0;
  if (cudaMemcpy(&e, err, 4, cudaMemcpyDeviceToHost) || cudaMemcpy(&b, bad, 8, cudaMemcpyDeviceToHost))
    return 6;
  printf("plans %d eight %d bad %llu err %d\n", plans, eight, b, e);
  return 0;
}
