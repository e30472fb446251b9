// Bias gradients of the decoder's linear layers: sums over the rows of a (rows, n) bf16 matrix, alone or while the gradient
// passes back through x sigmoid(x) (the feed-forward of flash_pop/retnet.py:247-268).
//
// Bound by HBM: one read of the matrix (and, with the activation, one more read and one write); the framework's reduction
// takes 18.6 us for 8192 x 1024 (16.8 MB, 0.9 TB/s), and the activation's backward was a pass of its own before it.  A warp
// takes 256 columns of a row, 16 bytes a lane, AHEAD rows in flight; the CTAs of a column tile share the rows (four CTAs an
// SM over all tiles, so a short matrix still covers the GPU) and leave fp32 partial sums in scratch memory, which a second
// launch, set up while the first drains, adds up in a fixed order: no zeroed accumulator, no atomic, the same result every
// time.  (Eight CTAs a tile that met in a cluster's shared memory read 128 bytes of a row at a time: 590 us for
// 262144 x 1024, where this takes 125 (4.3 TB/s) and 290 with the activation (5.6 TB/s); 8192 x 4096 with it 40 us.)
#include "fpb_common.cuh"

namespace fpb {
namespace {

typedef __nv_bfloat16 bf16;
constexpr int THREADS = 256, WARPS = 8, COLS = 256, MAX_SLABS = 148;

struct SumParams {
  const bf16* g; int64_t g_stride;                // (rows, n) gradient
  const bf16* a;                                  // ACT: (rows, n) contiguous input of the activation
  bf16* out;                                      // ACT: gradient of that input, contiguous
  float* partial;                                 // (slabs, n)
  bf16* sums;                                     // n
  int64_t rows;
  int32_t n, slabs;
};

// (volatile: left to itself the compiler moves each load down to its use, and the sums wait for one load at a time)
__device__ __forceinline__ uint4 ld_stream(const bf16* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}

template <bool ACT>
__global__ void __launch_bounds__(THREADS) column_sums_kernel(const __grid_constant__ SumParams p) {
  constexpr int AHEAD = ACT ? 4 : 8;
  __shared__ float part[WARPS][COLS + 4];
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, col = blockIdx.x * COLS + lane * 8;
  const int64_t step = (int64_t)p.slabs * WARPS, first = (int64_t)blockIdx.y * WARPS + warp;
  float acc[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) acc[e] = 0.0f;
  if (col < p.n) {
    for (int64_t r0 = first; r0 < p.rows; r0 += step * AHEAD) {
      uint4 g[AHEAD], a[ACT ? AHEAD : 1];
      // (rows past the end repeat the last one and are left out below: a load behind a branch would wait for the one before)
#pragma unroll
      for (int i = 0; i < AHEAD; ++i) {
        const int64_t r = min(r0 + i * step, p.rows - 1);
        g[i] = ld_stream(p.g + r * p.g_stride + col);
        if constexpr (ACT) a[i] = ld_stream(p.a + r * p.n + col);
      }
#pragma unroll
      for (int i = 0; i < AHEAD; ++i) {
        const int64_t r = r0 + i * step;
        if (r >= p.rows) break;
        const __nv_bfloat162* gv = reinterpret_cast<const __nv_bfloat162*>(&g[i]);
        uint4 res;
        __nv_bfloat162* rv = reinterpret_cast<__nv_bfloat162*>(&res);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          float2 f = __bfloat1622float2(gv[e]);
          if constexpr (ACT) {
            const float2 x = __bfloat1622float2(reinterpret_cast<const __nv_bfloat162*>(&a[i])[e]);
            const float sx = __fdividef(1.0f, 1.0f + __expf(-x.x)), sy = __fdividef(1.0f, 1.0f + __expf(-x.y));
            f.x *= sx * (1.0f + x.x * (1.0f - sx));
            f.y *= sy * (1.0f + x.y * (1.0f - sy));
            rv[e] = __float22bfloat162_rn(f);
          }
          acc[2 * e] += f.x; acc[2 * e + 1] += f.y;
        }
        if constexpr (ACT) *reinterpret_cast<uint4*>(p.out + r * p.n + col) = res;
      }
    }
  }
#pragma unroll
  for (int e = 0; e < 8; ++e) part[warp][lane * 8 + e] = acc[e];
  __syncthreads();
  const int c = blockIdx.x * COLS + threadIdx.x;
  float s = 0.0f;
#pragma unroll
  for (int w = 0; w < WARPS; ++w) s += part[w][threadIdx.x];
  if (c < p.n) p.partial[(int64_t)blockIdx.y * p.n + c] = s;
}

// 32 columns a CTA, a warp every eighth slab
__global__ void __launch_bounds__(THREADS) partial_sums_kernel(const __grid_constant__ SumParams p) {
  __shared__ float part[WARPS][33];
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, c = blockIdx.x * 32 + lane;
  float s = 0.0f;
#pragma unroll 4
  for (int k = warp; k < p.slabs; k += WARPS) s += p.partial[(int64_t)k * p.n + c];        // (n is a multiple of 64)
  part[warp][lane] = s;
  __syncthreads();
  if (warp == 0) {
#pragma unroll
    for (int w = 1; w < WARPS; ++w) s += part[w][lane];
    p.sums[c] = __float2bfloat16_rn(s);
  }
}

}  // namespace

int launch_column_sums(int64_t rows, int64_t n, const void* g, int64_t g_stride, const void* a, void* out, float* partial, void* sums,
                       cudaStream_t stream) {
  SumParams p{(const bf16*)g, g_stride, (const bf16*)a, (bf16*)out, partial, (bf16*)sums, rows, (int32_t)n, 1};
  const int tiles = (int)((n + COLS - 1) / COLS);
  int64_t slabs = FPB_COLUMN_SUMS_SCRATCH / 4 / n;                       // at most what the scratch holds: four CTAs an SM
  if (slabs > MAX_SLABS) slabs = MAX_SLABS;
  const int64_t most = (rows + WARPS * 4 - 1) / (WARPS * 4);             // four rows a warp at least
  p.slabs = (int)(slabs < most ? slabs : most);
  if (p.slabs < 1) p.slabs = 1;
  cudaError_t e = a ? launch_kernel(column_sums_kernel<true>, dim3(tiles, p.slabs), THREADS, 0, false, p, stream)
                    : launch_kernel(column_sums_kernel<false>, dim3(tiles, p.slabs), THREADS, 0, false, p, stream);
  if (e == cudaSuccess) e = launch_kernel(partial_sums_kernel, dim3((unsigned)(n / 32)), THREADS, 0, true, p, stream);
  return e == cudaSuccess ? FPB_OK : FPB_ERR_LAUNCH;
}

}  // namespace fpb
