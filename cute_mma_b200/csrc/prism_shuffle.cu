// Input shuffle folded into the parameters (reconn_sz 16, chunks of 64 features): the copies that put the columns of
// B_g, the internal bias and the rotation into physical feature order, and their adjoints for the gradients.
// A permutation never leaves its chunk and moves segments of two neighbouring features, so it is a table of 32 bytes per
// (group, chunk): segment i of the result is segment seg[i] of the source.  One warp owns one chunk of a row (one
// segment per lane): every row is read and written as whole 128-byte lines, whatever the permutation.
// Copies at memory speed: 4096 x 1024 bf16 (8.4 MB each way) 4.1 us; the gathers, scatters and stacks of torch that they
// replace were 8 launches of 11 us and about 30 small ones in a training step of that layer.
#include "../../include/prism_b200.h"
#include "prism_host.cuh"

namespace prism {

// T holds one segment: two 16-bit (uint32_t) or two 32-bit elements (uint2).
// Y[g*rows + r, 64 c + segment i] = X[g*rows + r, 64 c + segment seg[g, c, i]]
template <typename T>
__global__ void __launch_bounds__(256) shuffle_cols_kernel(const T* __restrict__ X, T* __restrict__ Y,
                                                           const uint8_t* __restrict__ seg, int n_chunks, int rows,
                                                           int rows_per_block) {
  const int lane = threadIdx.x & 31;
  const int c = blockIdx.x * 8 + (threadIdx.x >> 5);
  const int g = blockIdx.y;
  if (c >= n_chunks) return;
  const int src = seg[((long long)g * n_chunks + c) * 32 + lane] & 31;
  const long long pitch = (long long)n_chunks * 32;
  const int r0 = blockIdx.z * rows_per_block;
  const int n = min(rows_per_block, rows - r0);
  const long long base = ((long long)g * rows + r0) * pitch + c * 32;
  const T* x = X + base + src;
  T* y = Y + base + lane;
  int r = 0;
  for (; r + 8 <= n; r += 8) {   // eight rows in flight per warp
    T v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __ldg(x + (r + i) * pitch);
#pragma unroll
    for (int i = 0; i < 8; ++i) y[(r + i) * pitch] = v[i];
  }
  for (; r < n; ++r) y[r * pitch] = __ldg(x + r * pitch);
}

// R64[g*64 + i, 64 c + j] = bd[inv(i)][inv(j)] with bd = blockdiag of the chunk's four 16 x 16 blocks; seg: the inverse
// permutation (physical -> logical segment).  One warp per row of R64 and chunk.
__global__ void __launch_bounds__(256) shuffle_fold_r_kernel(const uint32_t* __restrict__ R, uint32_t* __restrict__ R64,
                                                             const uint8_t* __restrict__ seg, int n_chunks) {
  const int lane = threadIdx.x & 31;
  const int i = blockIdx.x * 8 + (threadIdx.x >> 5);   // 0..63: eight blocks of x
  const int c = blockIdx.y, g = blockIdx.z;
  const uint8_t* sg = seg + ((long long)g * n_chunks + c) * 32;
  const int a = (sg[i >> 1] & 31) * 2 + (i & 1);       // logical row of the chunk
  const int b = sg[lane] & 31;                         // logical segment (column pair)
  const long long pitch = (long long)n_chunks * 32;
  uint32_t v = 0;
  if ((a >> 4) == (b >> 3)) v = __ldg(R + ((long long)g * 16 + (a & 15)) * pitch + c * 32 + b);
  R64[((long long)g * 64 + i) * pitch + c * 32 + lane] = v;
}

// Adjoint: dR[g*16 + i, 64 c + j] = dR64[g*64 + perm(16 b + i), 64 c + perm(j)], b = j / 16; seg: the permutation
// (logical -> physical segment).  One warp per row of dR and chunk.
template <typename T>
__global__ void __launch_bounds__(256) shuffle_unfold_r_kernel(const T* __restrict__ D64, T* __restrict__ dR,
                                                               const uint8_t* __restrict__ seg, int n_chunks) {
  const int lane = threadIdx.x & 31;
  const int i = blockIdx.x * 8 + (threadIdx.x >> 5);   // 0..15: two blocks of x
  const int c = blockIdx.y, g = blockIdx.z;
  const uint8_t* sg = seg + ((long long)g * n_chunks + c) * 32;
  const int a = (lane >> 3) * 16 + i;                  // logical row of the block that this lane's column pair is in
  const int row = (sg[a >> 1] & 31) * 2 + (a & 1);
  const int col = sg[lane] & 31;
  const long long pitch = (long long)n_chunks * 32;
  dR[((long long)g * 16 + i) * pitch + c * 32 + lane] = __ldg(D64 + ((long long)g * 64 + row) * pitch + c * 32 + col);
}

static int check_shuffle(const char* fn, const void* in, const void* out, const void* seg, int G, int K, int esize) {
  if (in == nullptr || out == nullptr || seg == nullptr) return fail(PRISM_ERR_BAD_ARG, "%s: null pointer", fn);
  if (G <= 0 || G > 65535 || K <= 0 || K % 64 != 0 || K / 64 > 65535)
    return fail(PRISM_ERR_BAD_ARG, "%s: bad shape G=%d K=%d (K must be a multiple of 64)", fn, G, K);
  if (esize != 2 && esize != 4) return fail(PRISM_ERR_BAD_ARG, "%s: element size must be 2 or 4, got %d", fn, esize);
  if ((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out)) % (2 * esize) != 0)
    return fail(PRISM_ERR_BAD_ARG, "%s: matrices must be aligned to two elements", fn);
  return PRISM_OK;
}

}  // namespace prism

using namespace prism;

extern "C" int prism_shuffle_cols(const void* X, void* Y, const unsigned char* seg, int G, int rows_per_group, int K,
                                  int esize, void* stream) {
  const char* fn = "prism_shuffle_cols";
  int rc;
  if ((rc = check_shuffle(fn, X, Y, seg, G, K, esize))) return rc;
  if (rows_per_group <= 0) return fail(PRISM_ERR_BAD_ARG, "%s: rows_per_group must be positive", fn);
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  const int n_chunks = K / 64;
  int rpb = 32;   // rows per block: enough blocks to fill the GPU, eight rows in flight per warp
  while ((rows_per_group + rpb - 1) / rpb > 65535) rpb *= 2;
  const dim3 grid((n_chunks + 7) / 8, G, (rows_per_group + rpb - 1) / rpb);
  if (esize == 2)
    shuffle_cols_kernel<uint32_t><<<grid, 256, 0, s>>>(reinterpret_cast<const uint32_t*>(X), reinterpret_cast<uint32_t*>(Y),
                                                       seg, n_chunks, rows_per_group, rpb);
  else
    shuffle_cols_kernel<uint2><<<grid, 256, 0, s>>>(reinterpret_cast<const uint2*>(X), reinterpret_cast<uint2*>(Y), seg,
                                                    n_chunks, rows_per_group, rpb);
  return check_launch(fn);
}

extern "C" int prism_shuffle_fold_r(const void* R, void* R64, const unsigned char* inv_seg, int G, int K, void* stream) {
  const char* fn = "prism_shuffle_fold_r";
  int rc;
  if ((rc = check_shuffle(fn, R, R64, inv_seg, G, K, 2))) return rc;
  shuffle_fold_r_kernel<<<dim3(8, K / 64, G), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      reinterpret_cast<const uint32_t*>(R), reinterpret_cast<uint32_t*>(R64), inv_seg, K / 64);
  return check_launch(fn);
}

extern "C" int prism_shuffle_unfold_r(const void* dR64, void* dR, const unsigned char* seg, int G, int K, int esize,
                                      void* stream) {
  const char* fn = "prism_shuffle_unfold_r";
  int rc;
  if ((rc = check_shuffle(fn, dR64, dR, seg, G, K, esize))) return rc;
  const dim3 grid(2, K / 64, G);
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (esize == 2)
    shuffle_unfold_r_kernel<uint32_t><<<grid, 256, 0, s>>>(reinterpret_cast<const uint32_t*>(dR64),
                                                           reinterpret_cast<uint32_t*>(dR), seg, K / 64);
  else
    shuffle_unfold_r_kernel<uint2><<<grid, 256, 0, s>>>(reinterpret_cast<const uint2*>(dR64), reinterpret_cast<uint2*>(dR),
                                                        seg, K / 64);
  return check_launch(fn);
}
