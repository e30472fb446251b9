// One token through a stack of decoder layers (flash_pop/retnet.py:181-199,247-268: pre-norm, retention step, gate, output
// projection, feed-forward), five launches per layer, for batches of up to 64 rows:
//   1. project_kernel   LayerNorm of the row, then the q, k, v and gate projections
//   2. mix_kernel       rotation of q and k, S' = gamma S + k^T v / sqrt(dk), o = q S', GroupNorm of the head, gate
//   3. project_kernel   output projection + residual
//   4. project_kernel   LayerNorm, first feed-forward matrix, activation
//   5. project_kernel   second feed-forward matrix + residual
//
// What bounds it.  A token reads every weight and every state once and does next to no arithmetic, so the floor is HBM:
// 12 layers of d_model 1024, ffn 4096, 16 rows with fp32 states are 529 MB, 80 us at 6.65 TB/s.  As separate library and
// elementwise launches (20 a layer) the stack took 942 us on the device and 5900 us on the host.  A launch of one matrix
// is 1 to 8 MB, a microsecond of HBM time, so what counts is that every load of a launch is in flight at once and that no
// launch waits for its predecessor before it starts loading:
//   * a CTA owns NT weight rows over the whole contraction, its eight warps split K, and every warp requests its first
//     16 KB-a-warp of weights (16 x 16 bytes a thread: all there is for K <= 4096) before anything else;
//   * the launches are chained by programmatic dependent launch: weights and states, which no launch of the chain
//     writes, are requested before griddepcontrol.wait, i.e. while the predecessor is still running.  A kernel lets its
//     successor start only after its own wait, so whatever runs ahead of its wait has all launches but the last before
//     it behind it; every kernel waits, so the last one's end is the end of all.
// The products run on mma.sync.m16n8k16: rows of the batch x 8 weight rows, straight from the registers the 16-byte
// loads fill (the contraction index is permuted the same way in both operands: thread t of a quad holds elements
// 8t..8t+7 of every 32).  At 16 rows a weight byte feeds 16 multiply-adds, a hundredth of what tensor memory and
// tcgen05 tiles of 128 rows would pay for; their set-up would only add to the latency.
#include <atomic>

#include "fpb_common.cuh"

namespace fpb {
namespace {

typedef __nv_bfloat16 bf16;
constexpr int THREADS = 256, WARPS = 8;
constexpr int MAX_B = 64, MAX_D = 1024;          // rows of a batch; channels of a LayerNorm row (4 x 8 a lane)

__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ uint4 ld_stream(const void* p) {      // read once: keep it out of L1
  uint4 v;
  asm volatile("ld.global.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ void mma_16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float2 unpack2(uint32_t w) { return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w)); }
__device__ __forceinline__ uint32_t pack2(float a, float b) {
  const __nv_bfloat162 v = __float22bfloat162_rn(make_float2(a, b));
  return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ float activate(int kind, float x) {
  if (kind == FPB_ACT_SWISH) return __fdividef(x, 1.0f + __expf(-x));
  if (kind == FPB_ACT_GELU) return 0.5f * x * (1.0f + erff(x * 0.70710678118654752f));
  if (kind == FPB_ACT_RELU) return x < 0.0f ? 0.0f : x;          // (NaN passes)
  return x;
}

struct ProjectParams {
  const bf16* x; int64_t x_stride;               // (B, K) input rows
  const float *norm_w, *norm_b; float eps;       // LayerNorm of the rows (NORM launches); either may be null
  const bf16* w[4]; const bf16* bias[4];         // up to four (n_i, K) matrices whose outputs follow one another
  int32_t n_end[4];                              // last output + 1 of each
  const bf16* residual; int64_t res_stride;      // added to the (bf16-rounded) projection, or null
  bf16* y; int64_t y_stride;
  int32_t B, K, act;
};

__host__ __device__ constexpr int norm_pitch(int K) { return K * 2 + 64; }   // bytes: eight rows x four 16-byte pieces of a quad tile all 32 banks

// N8: weight rows a CTA owns / 8; MT: batch rows / 16, rounded up.
template <int N8, int MT, bool NORM>
__global__ void __launch_bounds__(THREADS, MT <= 2 ? 2 : 1) project_kernel(const __grid_constant__ ProjectParams p) {
  constexpr int NT = N8 * 8, BLK = 16 / N8;      // BLK: 32-wide contraction steps whose weights are in flight together
  extern __shared__ __align__(16) uint8_t sm[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int n0 = blockIdx.x * NT;
  int m = 0;
#pragma unroll
  for (int i = 0; i < 3; ++i) m += n0 >= p.n_end[i] ? 1 : 0;
  const int n_first = n0 - (m ? p.n_end[m - 1] : 0);
  const int K = p.K, steps = K >> 5;
  const int i0 = steps * warp / WARPS, i1 = steps * (warp + 1) / WARPS;
  const bf16* w = p.w[m] + (int64_t)(n_first + g) * K + t * 8;

  uint4 wr[BLK][N8];
  auto fetch = [&](int base) {
#pragma unroll
    for (int j = 0; j < BLK; ++j)
#pragma unroll
      for (int c = 0; c < N8; ++c)
        if (base + j < i1) wr[j][c] = ld_stream(w + (int64_t)c * 8 * K + (base + j) * 32);
  };
  fetch(i0);
  grid_wait();
  grid_release();

  const int pitch = norm_pitch(K);
  if constexpr (NORM) {                           // normalised rows, rounded to bf16 as the operand of the products
    for (int row = warp; row < p.B; row += WARPS) {
      const bf16* x = p.x + row * p.x_stride;
      float f[4][8];
      float sum = 0.0f;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int c = 8 * (lane + 32 * i);
        if (c < K) {
          const uint4 raw = *reinterpret_cast<const uint4*>(x + c);
          const uint32_t e[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
          for (int j = 0; j < 4; ++j) { const float2 a = unpack2(e[j]); f[i][2 * j] = a.x; f[i][2 * j + 1] = a.y; sum += a.x + a.y; }
        }
      }
      const float mean = warp_sum(sum) / (float)K;
      float sq = 0.0f;
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (8 * (lane + 32 * i) < K) {
#pragma unroll
          for (int j = 0; j < 8; ++j) { f[i][j] -= mean; sq += f[i][j] * f[i][j]; }
        }
      const float rstd = rsqrtf(warp_sum(sq) / (float)K + p.eps);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int c = 8 * (lane + 32 * i);
        if (c < K) {
          uint32_t e[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float2 gw = p.norm_w ? __ldg(reinterpret_cast<const float2*>(p.norm_w + c) + j) : make_float2(1.0f, 1.0f);
            const float2 gb = p.norm_b ? __ldg(reinterpret_cast<const float2*>(p.norm_b + c) + j) : make_float2(0.0f, 0.0f);
            e[j] = pack2(f[i][2 * j] * rstd * gw.x + gb.x, f[i][2 * j + 1] * rstd * gw.y + gb.y);
          }
          *reinterpret_cast<uint4*>(sm + row * pitch + c * 2) = make_uint4(e[0], e[1], e[2], e[3]);
        }
      }
    }
    __syncthreads();
  }

  float acc[MT][N8][4];
#pragma unroll
  for (int a = 0; a < MT; ++a)
#pragma unroll
    for (int c = 0; c < N8; ++c)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[a][c][e] = 0.0f;
  // rows past the batch repeat its last row; their sums are dropped
  auto x_piece = [&](int row, int step) -> uint4 {
    row = min(row, p.B - 1);
    if constexpr (NORM) return *reinterpret_cast<const uint4*>(sm + row * pitch + (step * 32 + t * 8) * 2);
    else return *reinterpret_cast<const uint4*>(p.x + row * p.x_stride + step * 32 + t * 8);
  };
  constexpr int XB = MT == 1 ? 4 : MT == 2 ? 2 : 1;        // steps whose inputs are in flight together
  for (int base = i0; base < i1; base += BLK) {
#pragma unroll
    for (int j0 = 0; j0 < BLK; j0 += XB) {
      uint4 lo[XB][MT], hi[XB][MT];
#pragma unroll
      for (int j = 0; j < XB; ++j)
#pragma unroll
        for (int a = 0; a < MT; ++a) {
          const int step = min(base + j0 + j, i1 - 1);
          lo[j][a] = x_piece(a * 16 + g, step);
          hi[j][a] = x_piece(a * 16 + g + 8, step);
        }
#pragma unroll
      for (int j = 0; j < XB; ++j) {
        if (base + j0 + j >= i1) break;
#pragma unroll
        for (int a = 0; a < MT; ++a)
#pragma unroll
          for (int c = 0; c < N8; ++c) {
            const uint4 b = wr[j0 + j][c];
            mma_16816(acc[a][c], lo[j][a].x, hi[j][a].x, lo[j][a].y, hi[j][a].y, b.x, b.y);
            mma_16816(acc[a][c], lo[j][a].z, hi[j][a].z, lo[j][a].w, hi[j][a].w, b.z, b.w);
          }
      }
    }
    fetch(base + BLK);
  }

  // the warps' partial sums over K
  float* red = reinterpret_cast<float*>(sm + (NORM ? MT * 16 * pitch : 0));   // [WARPS][MT * 16][NT + 2]
  constexpr int RP = NT + 2;
#pragma unroll
  for (int a = 0; a < MT; ++a)
#pragma unroll
    for (int c = 0; c < N8; ++c) {
      float* r = red + ((warp * MT + a) * 16 + g) * RP + c * 8 + 2 * t;
      *reinterpret_cast<float2*>(r) = make_float2(acc[a][c][0], acc[a][c][1]);
      *reinterpret_cast<float2*>(r + 8 * RP) = make_float2(acc[a][c][2], acc[a][c][3]);
    }
  __syncthreads();
  for (int idx = threadIdx.x; idx < p.B * (NT / 2); idx += THREADS) {
    const int row = idx / (NT / 2), c = (idx % (NT / 2)) * 2;
    float2 s = make_float2(0.0f, 0.0f);
#pragma unroll
    for (int k = 0; k < WARPS; ++k) {
      const float2 v = *reinterpret_cast<const float2*>(red + (k * MT * 16 + row) * RP + c);
      s.x += v.x; s.y += v.y;
    }
    if (p.bias[m]) {
      const float2 b = unpack2(*reinterpret_cast<const uint32_t*>(p.bias[m] + n_first + c));
      s.x += b.x; s.y += b.y;
    }
    s.x = activate(p.act, s.x); s.y = activate(p.act, s.y);
    uint32_t out = pack2(s.x, s.y);
    if (p.residual) {
      const float2 y = unpack2(out), r = unpack2(*reinterpret_cast<const uint32_t*>(p.residual + row * p.res_stride + n0 + c));
      out = pack2(r.x + y.x, r.y + y.y);
    }
    *reinterpret_cast<uint32_t*>(p.y + row * p.y_stride + n0 + c) = out;
  }
}

struct MixParams {
  const bf16* qkvg;                               // (B, 2 H dk + 2 H dv): q | k | v | gate
  const float2* phasors;                          // (dk / 2) of (cos, sin) for this position, or null
  const void* s_prev; int64_t prev_sb, prev_sh;   // null: a zero state
  void* s_out; int64_t out_sb, out_sh;
  bf16* y;                                        // (B, H dv)
  int32_t H, dk, dv, act;
  float gn_eps;
  float gamma[FPB_MAX_HEADS];
};

template <typename T> __device__ __forceinline__ float4 load4(const T* p);
template <> __device__ __forceinline__ float4 load4<float>(const float* p) { return *reinterpret_cast<const float4*>(p); }
template <> __device__ __forceinline__ float4 load4<bf16>(const bf16* p) {
  const uint2 r = *reinterpret_cast<const uint2*>(p);
  const float2 a = unpack2(r.x), b = unpack2(r.y);
  return make_float4(a.x, a.y, b.x, b.y);
}
template <typename T> __device__ __forceinline__ void store4(T* p, float4 v);
template <> __device__ __forceinline__ void store4<float>(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
template <> __device__ __forceinline__ void store4<bf16>(bf16* p, float4 v) { *reinterpret_cast<uint2*>(p) = make_uint2(pack2(v.x, v.y), pack2(v.z, v.w)); }

// A CTA owns one (row, head): dv / 4 threads across the state's columns, as many rows at a time as the 256 threads hold,
// eight passes of rows in flight while the eight before them are worked on.
template <typename TP, typename TO>
__global__ void __launch_bounds__(THREADS, 2) mix_kernel(const __grid_constant__ MixParams p) {
  constexpr int UN = 8;
  __shared__ float sh_q[256], sh_k[256], sh_red[2][WARPS];
  __shared__ float sh_o[THREADS * 4];
  const int h = blockIdx.x, b = blockIdx.y, tid = threadIdx.x;
  const int tx_n = p.dv >> 2, ty_n = THREADS / tx_n;
  const int tx = tid % tx_n, ty = tid / tx_n, col = tx * 4;
  const bool live = ty < ty_n;
  const TP* sp = p.s_prev && live ? (const TP*)p.s_prev + b * p.prev_sb + h * p.prev_sh + col : nullptr;
  TO* so = (TO*)p.s_out + b * p.out_sb + h * p.out_sh + col;
  const float gamma = p.gamma[h];

  float4 ra[UN], rb[UN];
  auto fetch = [&](float4 (&r)[UN], int r0) {
#pragma unroll
    for (int u = 0; u < UN; ++u) {
      const int row = r0 + u * ty_n;
      r[u] = sp && row < p.dk ? load4<TP>(sp + (int64_t)row * p.dv) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  };
  fetch(ra, ty);
  grid_wait();
  grid_release();

  const int qk = p.H * p.dk, width = p.H * p.dv;
  const bf16* in = p.qkvg + (int64_t)b * (2 * qk + 2 * width);
  const float rs = rsqrtf((float)p.dk);
  for (int i = tid; i < p.dk / 2; i += THREADS) {
    float2 q = unpack2(*reinterpret_cast<const uint32_t*>(in + h * p.dk + 2 * i));
    float2 k = unpack2(*reinterpret_cast<const uint32_t*>(in + qk + h * p.dk + 2 * i));
    if (p.phasors) {
      const float2 c = p.phasors[i];
      q = make_float2(q.x * c.x - q.y * c.y, q.x * c.y + q.y * c.x);
      k = make_float2(k.x * c.x - k.y * c.y, k.x * c.y + k.y * c.x);
    }
    sh_q[2 * i] = q.x; sh_q[2 * i + 1] = q.y;
    sh_k[2 * i] = k.x * rs; sh_k[2 * i + 1] = k.y * rs;
  }
  const float4 v = live ? load4<bf16>(in + 2 * qk + h * p.dv + col) : make_float4(0.f, 0.f, 0.f, 0.f);
  const float z = tid < p.dv ? __bfloat162float(in[2 * qk + width + h * p.dv + tid]) : 0.0f;
  __syncthreads();
  float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
  auto update = [&](const float4 (&r)[UN], int r0) {
#pragma unroll
    for (int u = 0; u < UN; ++u) {
      const int row = r0 + u * ty_n;
      if (live && row < p.dk) {
        const float kr = sh_k[row], qr = sh_q[row];
        float4 s;
        s.x = fmaf(gamma, r[u].x, kr * v.x); s.y = fmaf(gamma, r[u].y, kr * v.y);
        s.z = fmaf(gamma, r[u].z, kr * v.z); s.w = fmaf(gamma, r[u].w, kr * v.w);
        o.x = fmaf(qr, s.x, o.x); o.y = fmaf(qr, s.y, o.y); o.z = fmaf(qr, s.z, o.z); o.w = fmaf(qr, s.w, o.w);
        store4<TO>(so + (int64_t)row * p.dv, s);
      }
    }
  };
  const int pass = UN * ty_n;
  for (int r0 = ty; r0 < p.dk; r0 += 2 * pass) {
    fetch(rb, r0 + pass);
    update(ra, r0);
    fetch(ra, r0 + 2 * pass);
    update(rb, r0 + pass);
  }
  if (live) *reinterpret_cast<float4*>(sh_o + ty * p.dv + col) = o;
  __syncthreads();
  float x = 0.0f;
  if (tid < p.dv)
    for (int y = 0; y < ty_n; ++y) x += sh_o[y * p.dv + tid];
  // GroupNorm over the head's dv outputs, one a thread
  auto block_sum = [&](float f, int buf) {
    f = warp_sum(f);
    if ((tid & 31) == 0) sh_red[buf][tid >> 5] = f;
    __syncthreads();
    float s = 0.0f;
#pragma unroll
    for (int i = 0; i < WARPS; ++i) s += sh_red[buf][i];
    return s;
  };
  const float mean = block_sum(x, 0) / (float)p.dv;
  const float d = tid < p.dv ? x - mean : 0.0f;
  const float rstd = rsqrtf(block_sum(d * d, 1) / (float)p.dv + p.gn_eps);
  if (tid < p.dv) p.y[(int64_t)b * width + h * p.dv + tid] = __float2bfloat16_rn(d * rstd * activate(p.act, z));
}

// Launch with (or, for the first of a chain, without) permission to start before the launch ahead of it has ended.
template <typename P>
cudaError_t launch(void (*kernel)(P), dim3 grid, size_t smem, bool chained, const P& p, cudaStream_t stream) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid; cfg.blockDim = dim3(THREADS); cfg.dynamicSmemBytes = smem; cfg.stream = stream;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr; cfg.numAttrs = chained ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, p);
}

template <int N8, int MT, bool NORM>
cudaError_t launch_project_t(const ProjectParams& p, int n, bool chained, cudaStream_t stream) {
  constexpr int RED = WARPS * MT * 16 * (N8 * 8 + 2) * 4;
  constexpr int MOST = (NORM ? MT * 16 * norm_pitch(MAX_D) : 0) + RED;
  static_assert(MOST <= 227 * 1024, "shared memory of a CTA");
  static std::atomic<bool> configured[64];
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64 || !configured[dev].load(std::memory_order_acquire)) {
    const cudaError_t e = cudaFuncSetAttribute(project_kernel<N8, MT, NORM>, cudaFuncAttributeMaxDynamicSharedMemorySize, MOST);
    if (e != cudaSuccess) return e;
    if (dev >= 0 && dev < 64) configured[dev].store(true, std::memory_order_release);
  }
  const size_t smem = (NORM ? MT * 16 * norm_pitch(p.K) : 0) + RED;
  return launch(project_kernel<N8, MT, NORM>, dim3(n / (N8 * 8)), smem, chained, p, stream);
}

// Rows a CTA owns: as few as still make one CTA an SM or so (128 CTAs for 1024 to 4096 outputs), which spreads a small
// matrix over the GPU; 32 at most, which is what the registers hold.  Every matrix of the launch is a multiple of them.
template <int MT, bool NORM>
cudaError_t launch_project_m(const ProjectParams& p, int n, bool chained, cudaStream_t stream) {
  auto fits = [&](int nt) {
    for (int i = 0; i < 4; ++i)
      if (p.n_end[i] % nt) return false;
    return true;
  };
  if (n > 2 * 8 * 148 && fits(32)) return launch_project_t<4, MT, NORM>(p, n, chained, stream);
  if (n > 8 * 148 && fits(16)) return launch_project_t<2, MT, NORM>(p, n, chained, stream);
  return launch_project_t<1, MT, NORM>(p, n, chained, stream);
}
template <bool NORM>
cudaError_t launch_project(const ProjectParams& p, int n, bool chained, cudaStream_t stream) {
  if (p.B <= 16) return launch_project_m<1, NORM>(p, n, chained, stream);
  if (p.B <= 32) return launch_project_m<2, NORM>(p, n, chained, stream);
  return launch_project_m<4, NORM>(p, n, chained, stream);
}

bool aligned(const void* p, int n) { return (uintptr_t)p % n == 0; }

}  // namespace

int64_t decoder_token_workspace(const fpb_token_dims& d) {
  const int64_t qk = (int64_t)d.H * d.dk, width = (int64_t)d.H * d.dv;
  return 2 * (int64_t)d.B * (2 * qk + 2 * width + 3 * width + d.ffn) + 64;     // qkvg | gated | two streams of x | ffn, bf16
}

int check_decoder_token(const fpb_token_dims& d, const fpb_decoder_layer* layers) {
  if (d.layers < 0 || d.B < 0 || d.H <= 0 || d.dk <= 0 || d.dv <= 0 || d.ffn <= 0) return FPB_ERR_BAD_SHAPE;
  const int64_t width = (int64_t)d.H * d.dv, qk = (int64_t)d.H * d.dk;
  if (d.H > FPB_MAX_HEADS || d.dk > 256 || d.dv > 256 || d.B > MAX_B || width > MAX_D || d.ffn > (1 << 20) || qk > (1 << 20)) return FPB_ERR_BAD_SHAPE;
  if (d.dk % 2 || d.dv % 4 || width % 32 || qk % 8 || d.ffn % 32) return FPB_ERR_BAD_SHAPE;
  if ((d.prev_dtype != FPB_BF16 && d.prev_dtype != FPB_F32) || (d.out_dtype != FPB_BF16 && d.out_dtype != FPB_F32)) return FPB_ERR_BAD_DTYPE;
  if (d.layers == 0 || d.B == 0) return FPB_OK;
  if (!layers || !d.head_decays || !d.workspace) return FPB_ERR_NULL_POINTER;
  if (!aligned(d.workspace, 16) || d.workspace_bytes < decoder_token_workspace(d)) return FPB_ERR_BAD_WORKSPACE;
  const int64_t blk = (int64_t)d.dk * d.dv;
  for (int i = 0; i < d.layers; ++i) {
    const fpb_decoder_layer& l = layers[i];
    for (const void* w : {l.wq, l.wk, l.wv, l.wg, l.wo, l.w1, l.w2}) {
      if (!w) return FPB_ERR_NULL_POINTER;
      if (!aligned(w, 16)) return FPB_ERR_BAD_STRIDE;
    }
    for (const void* b : {l.bq, l.bk, l.bv, l.bg, l.bo, l.b1, l.b2})
      if (!aligned(b, 4)) return FPB_ERR_BAD_STRIDE;
    for (const float* v : {l.norm1_w, l.norm1_b, l.norm2_w, l.norm2_b, l.phasors})
      if (!aligned(v, 8)) return FPB_ERR_BAD_STRIDE;
    if (l.act_gate < 0 || l.act_gate > FPB_ACT_RELU || l.act_ffn < 0 || l.act_ffn > FPB_ACT_RELU) return FPB_ERR_BAD_SHAPE;
    if (!l.s_out) return FPB_ERR_NULL_POINTER;
    // rows of four state elements are read and written at a time
    if (!aligned(l.s_out, d.out_dtype == FPB_F32 ? 16 : 8) || l.out_sb % 4 || l.out_sh % 4) return FPB_ERR_BAD_STRIDE;
    if (!aligned(l.s_prev, d.prev_dtype == FPB_F32 ? 16 : 8) || l.prev_sb % 4 || l.prev_sh % 4) return FPB_ERR_BAD_STRIDE;
    if ((d.H > 1 && l.out_sh < blk) || (d.B > 1 && l.out_sb < blk)) return FPB_ERR_BAD_STRIDE;
    if (l.s_prev && ((d.H > 1 && l.prev_sh < blk) || (d.B > 1 && l.prev_sb < blk))) return FPB_ERR_BAD_STRIDE;
  }
  return FPB_OK;
}

int launch_decoder_token(const fpb_token_dims& d, const fpb_decoder_layer* layers, const float* gamma, const void* x, int64_t x_stride,
                         void* y, int64_t y_stride, cudaStream_t stream, int* n_launched) {
  const int width = d.H * d.dv, qk = d.H * d.dk, n4 = 2 * qk + 2 * width;
  bf16* buf = (bf16*)d.workspace;
  auto take = [&](int64_t n) { bf16* r = buf; buf += (n + 7) / 8 * 8; return r; };
  bf16* qkvg = take((int64_t)d.B * n4);
  bf16* gated = take((int64_t)d.B * width);
  bf16* mid = take((int64_t)d.B * width);         // x + retention of the layer
  bf16* stream_x = take((int64_t)d.B * width);    // x between layers
  bf16* hidden = take((int64_t)d.B * d.ffn);
  const bf16* in = (const bf16*)x; int64_t in_stride = x_stride;
  bool chained = false;
  cudaError_t e = cudaSuccess;
  for (int i = 0; i < d.layers && e == cudaSuccess; ++i) {
    const fpb_decoder_layer& l = layers[i];
    ProjectParams p{};
    p.B = d.B; p.K = width; p.act = FPB_ACT_NONE;
    p.x = in; p.x_stride = in_stride; p.norm_w = l.norm1_w; p.norm_b = l.norm1_b; p.eps = (float)l.norm1_eps;
    p.w[0] = (const bf16*)l.wq; p.w[1] = (const bf16*)l.wk; p.w[2] = (const bf16*)l.wv; p.w[3] = (const bf16*)l.wg;
    p.bias[0] = (const bf16*)l.bq; p.bias[1] = (const bf16*)l.bk; p.bias[2] = (const bf16*)l.bv; p.bias[3] = (const bf16*)l.bg;
    p.n_end[0] = qk; p.n_end[1] = 2 * qk; p.n_end[2] = 2 * qk + width; p.n_end[3] = n4;
    p.y = qkvg; p.y_stride = n4;
    if ((e = launch_project<true>(p, n4, chained, stream)) != cudaSuccess) break;
    chained = true;

    MixParams mx;
    mx.qkvg = qkvg; mx.phasors = (const float2*)l.phasors;
    mx.s_prev = l.s_prev; mx.prev_sb = l.prev_sb; mx.prev_sh = l.prev_sh;
    mx.s_out = l.s_out; mx.out_sb = l.out_sb; mx.out_sh = l.out_sh;
    mx.y = gated; mx.H = d.H; mx.dk = d.dk; mx.dv = d.dv; mx.act = (int)l.act_gate; mx.gn_eps = (float)l.gn_eps;
    for (int h = 0; h < d.H; ++h) mx.gamma[h] = gamma[h];
    const dim3 mgrid(d.H, d.B);
    if (d.out_dtype == FPB_F32)
      e = d.prev_dtype == FPB_F32 ? launch(mix_kernel<float, float>, mgrid, 0, true, mx, stream) : launch(mix_kernel<bf16, float>, mgrid, 0, true, mx, stream);
    else
      e = d.prev_dtype == FPB_F32 ? launch(mix_kernel<float, bf16>, mgrid, 0, true, mx, stream) : launch(mix_kernel<bf16, bf16>, mgrid, 0, true, mx, stream);
    if (e != cudaSuccess) break;

    auto one = [&](const bf16* src, int K, const void* w, const void* b, int n) {      // a launch of one matrix
      ProjectParams r{};
      r.B = d.B; r.K = K; r.act = FPB_ACT_NONE; r.x = src; r.x_stride = K;
      r.w[0] = (const bf16*)w; r.bias[0] = (const bf16*)b;
      for (int j = 0; j < 4; ++j) r.n_end[j] = n;
      return r;
    };
    ProjectParams po = one(gated, width, l.wo, l.bo, width);
    po.residual = in; po.res_stride = in_stride; po.y = mid; po.y_stride = width;
    if ((e = launch_project<false>(po, width, true, stream)) != cudaSuccess) break;
    ProjectParams p1 = one(mid, width, l.w1, l.b1, d.ffn);
    p1.norm_w = l.norm2_w; p1.norm_b = l.norm2_b; p1.eps = (float)l.norm2_eps; p1.act = (int)l.act_ffn;
    p1.y = hidden; p1.y_stride = d.ffn;
    if ((e = launch_project<true>(p1, d.ffn, true, stream)) != cudaSuccess) break;
    ProjectParams p2 = one(hidden, d.ffn, l.w2, l.b2, width);
    const bool last = i == d.layers - 1;
    p2.residual = mid; p2.res_stride = width; p2.y = last ? (bf16*)y : stream_x; p2.y_stride = last ? y_stride : width;
    e = launch_project<false>(p2, width, true, stream);
    in = stream_x; in_stride = width;
    *n_launched += 5;
  }
  return e == cudaSuccess ? FPB_OK : FPB_ERR_LAUNCH;
}

}  // namespace fpb
