// One token through a stack of decoder layers (flash_pop/retnet.py:181-199,247-268: pre-norm, retention step, gate, output
// projection, feed-forward) in one cooperative launch, for batches of up to 64 rows.  Per layer five phases, a grid
// barrier after each:
//   0. LayerNorm of the rows, then the q, k, v and gate projections
//   1. rotation of q and k, S' = gamma S + k^T v / sqrt(dk), o = q S', GroupNorm of the head, gate
//   2. output projection + residual
//   3. LayerNorm, first feed-forward matrix, activation
//   4. second feed-forward matrix + residual
//
// What bounds it.  A token reads every weight and every state once and does next to no arithmetic, so the floor is HBM:
// 12 layers of d_model 1024, ffn 4096, 16 rows with fp32 states are 529 MB, 80 us at 6.65 TB/s, a microsecond a phase.
// What a phase costs beyond that is latency: of its first loads and of the hand-over from the phase before.  So
//   * weights and states are requested into L2 two phases ahead, and every thread loads its first 128 bytes of the next
//     phase's, with its bias and norm parameters, before it arrives at the barrier - no phase writes any of them - so HBM
//     streams while the grid synchronises;
//   * a phase deals its weight rows out in eights, evenly over the SMs, and the 16 warps of a CTA split the contraction;
//   * up to 16 rows each CTA normalises the rows it reads itself, one warp a row; beyond, 128 KB of rows read and normalised
//     by every SM cost more (38000 cycles at 64 rows) than a phase of its own that does it once.
// Measured (12 layers as above, device time by graph replay / with the host work): 241 library and elementwise launches
// 942 / 5870 us, five launches a layer chained by programmatic dependent launch 395 / 422 us, one launch 372 / 374 us (1 row
// 332, 32 rows 489, 64 rows 801; the chained launches took 895 at 64).  A phase is 7000 to 13000 cycles, 2000 of them the
// barrier; the rest is dependent round trips to L2 (700 to 1000 cycles each) and straight-line code run once.
//
// The products run on mma.sync.m16n8k16: rows of the batch x 8 weight rows, straight from the registers the 16-byte
// loads fill (the contraction index is permuted the same way in both operands: thread t of a quad holds elements
// 8t..8t+7 of every 32).  At 16 rows a weight byte feeds 16 multiply-adds, a hundredth of what tensor memory and
// tcgen05 tiles of 128 rows would pay for; their set-up would only add to the latency.
#include <atomic>

#include "fpb_common.cuh"

namespace fpb {
namespace {

typedef __nv_bfloat16 bf16;
constexpr int THREADS = 512, WARPS = 16;
// Rows of a batch and channels of a LayerNorm row.  Neither is a limit of the machine: 64 rows are four 16-row tiles of
// accumulators a warp (MT = 4, the largest instance built), 1024 channels what normalise() keeps in a lane's registers, what
// is staged of a norm's parameters, and what the library's LayerNorm takes of bf16 rows.  Beyond either the layers run one by
// one, which costs their host work whatever the size: 12 layers of d_model 1024, 64 rows here 870 us a call, 65 rows 3990;
// d_model 2048, 16 rows 4350.
constexpr int MAX_B = 64, MAX_D = 1024;
constexpr int MAX_LAYERS = 16;                   // of a launch (the layers' records are kernel parameters)
constexpr int PF = 8;                            // 16-byte pieces a thread has in flight

struct TokenParams {
  int32_t B, H, dk, dv, ffn, layers, prev_f32, out_f32;
  const bf16* x; int64_t x_stride;
  bf16* y; int64_t y_stride;
  bf16 *qkvg, *gated, *mid, *between, *hidden, *normed;   // (B, 2 H dk + 2 H dv), (B, H dv) three times, (B, ffn), (B, H dv)
  unsigned* arrived;                              // the grid barrier's count, zero at the start
  int32_t* status;
  long long wait_cycles;
  float gamma[FPB_MAX_HEADS];
  fpb_decoder_layer layer[MAX_LAYERS];
};

__device__ __forceinline__ uint4 ld_stream(const void* p) {      // read once: keep it out of L1
  uint4 v;
  asm volatile("ld.global.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ unsigned ld_acquire(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void add_release(unsigned* p) {
  asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(p) : "memory");
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
// What other CTAs wrote during this launch is read past L1, which nothing keeps coherent.
__device__ __forceinline__ uint4 ld_fresh(const void* p) { return __ldcg(reinterpret_cast<const uint4*>(p)); }

// One projection phase: y = x W^T with up to four matrices whose outputs follow one another.  Kept in shared memory: made
// anew from the kernel's parameters in every phase it cost 800 cycles each time (constant-cache misses).
struct Job {
  const void* w[4]; const void* bias[4];
  int32_t n_beg[4], n_end[4];                     // first output of each and last + 1
  int32_t N, K, act;
  const float *norm_w, *norm_b; float eps;        // phases 0 and 3
  const bf16* in; int64_t in_stride;              // rows that the norm reads
  const bf16* x; int64_t x_stride;                // rows that the products read: the same, or their norms
  const bf16* residual; int64_t res_stride;
  bf16* y; int64_t y_stride;
};

__host__ __device__ constexpr int norm_pitch(int K) { return K * 2 + 64; }   // bytes: eight rows x a quad's pieces tile all banks

__device__ __forceinline__ Job job_of(const TokenParams& p, int i, int phase, bool normed) {
  const fpb_decoder_layer& l = p.layer[i];
  const int width = p.H * p.dv, qk = p.H * p.dk;
  const bf16* in = i == 0 ? p.x : p.between;
  const int64_t in_stride = i == 0 ? p.x_stride : width;
  Job j{};
  j.act = FPB_ACT_NONE;
  if (phase == 0) {
    j.w[0] = l.wq; j.w[1] = l.wk; j.w[2] = l.wv; j.w[3] = l.wg;
    j.bias[0] = l.bq; j.bias[1] = l.bk; j.bias[2] = l.bv; j.bias[3] = l.bg;
    j.n_end[0] = qk; j.n_end[1] = 2 * qk; j.n_end[2] = 2 * qk + width; j.n_end[3] = 2 * qk + 2 * width;
    j.K = width; j.norm_w = l.norm1_w; j.norm_b = l.norm1_b; j.eps = (float)l.norm1_eps;
    j.x = in; j.x_stride = in_stride; j.y = p.qkvg; j.y_stride = j.n_end[3];
  } else {
    j.w[0] = phase == 2 ? l.wo : phase == 3 ? l.w1 : l.w2;
    j.bias[0] = phase == 2 ? l.bo : phase == 3 ? l.b1 : l.b2;
    const int n = phase == 3 ? p.ffn : width;
    j.n_end[0] = j.n_end[1] = j.n_end[2] = j.n_end[3] = n;
    j.K = phase == 4 ? p.ffn : width;
    j.x = phase == 2 ? p.gated : phase == 3 ? p.mid : p.hidden; j.x_stride = j.K;
    j.y = phase == 2 ? p.mid : phase == 3 ? p.hidden : p.between; j.y_stride = n;
    if (phase == 2) { j.residual = in; j.res_stride = in_stride; }
    if (phase == 3) { j.norm_w = l.norm2_w; j.norm_b = l.norm2_b; j.eps = (float)l.norm2_eps; j.act = (int)l.act_ffn; }
    if (phase == 4) {
      j.residual = p.mid; j.res_stride = width;
      if (i == p.layers - 1) { j.y = p.y; j.y_stride = p.y_stride; }
    }
  }
  j.in = j.x; j.in_stride = j.x_stride;
  if (normed && (phase == 0 || phase == 3)) { j.x = p.normed; j.x_stride = width; }
  j.n_beg[0] = 0; j.n_beg[1] = j.n_end[0]; j.n_beg[2] = j.n_end[1]; j.n_beg[3] = j.n_end[2];
  j.N = j.n_end[3];
  return j;
}

struct Share { int c0, c1, k0, k1; };             // weight rows / 8 of this CTA; 32-wide contraction steps of this warp
__device__ __forceinline__ Share share_of(const Job& j, const int2& tiles) {
  const int steps = j.K >> 5, warp = threadIdx.x >> 5;
  return {tiles.x, tiles.y, steps * warp / WARPS, steps * (warp + 1) / WARPS};
}
__device__ __forceinline__ void prefetch_l2(const void* p, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copy_async16(void* smem, const void* p) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(p) : "memory");
}
__device__ __forceinline__ void copy_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }
__device__ __forceinline__ int matrix_of(const Job& j, int n0) {
  int m = 0;
#pragma unroll
  for (int i = 0; i < 3; ++i) m += n0 >= j.n_end[i] ? 1 : 0;
  return m;
}
// this thread's pieces of weight tiles [tile, tile + TPP), steps [step, step + PF / TPP)
template <int TPP> __device__ __forceinline__ void fetch_weights(uint4 (&w)[PF], const Job& j, const Share& s, int tile, int step) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int c = 0; c < TPP; ++c) {
    const int n0 = (tile + c) * 8, m = matrix_of(j, n0);
    const bf16* base = (const bf16*)j.w[m] + (int64_t)(n0 - j.n_beg[m] + g) * j.K + t * 8;
#pragma unroll
    for (int i = 0; i < PF / TPP; ++i)
      if (tile + c < s.c1 && step + i < s.k1) w[i * TPP + c] = ld_stream(base + (step + i) * 32);
  }
}

// the bias of the column pair this thread finishes
template <int TPP> __device__ __forceinline__ uint32_t fetch_bias(const Job& j, const Share& s, int tile) {
  const int n = tile * 8 + (threadIdx.x % (TPP * 4)) * 2, m = matrix_of(j, n);
  const bf16* bias = (const bf16*)j.bias[m];
  return bias && n < s.c1 * 8 ? __ldg(reinterpret_cast<const unsigned*>(bias + n - j.n_beg[m])) : 0u;
}

// the norm's weight and bias, MAX_D floats each, into shared memory ahead of the barrier
__device__ __forceinline__ void stage_norm(float* dst, const Job& j) {
  const int i = (threadIdx.x & 255) * 4;
  const float* src = threadIdx.x < 256 ? j.norm_w : j.norm_b;
  float* to = dst + (threadIdx.x < 256 ? 0 : MAX_D) + i;
  if (i >= j.K) return;
  const float fill = threadIdx.x < 256 ? 1.0f : 0.0f;
  if (src) copy_async16(to, src + i);
  else *reinterpret_cast<float4*>(to) = make_float4(fill, fill, fill, fill);
}
static_assert(THREADS == 512 && MAX_D == 1024, "one 16-byte piece a thread");

// LayerNorm of the batch's rows, rounded to bf16 as the operand of the products: a warp a row, its next row on its way.  Four channels a lane and piece: the parameters' 16-byte loads then meet no bank conflict.
__device__ __forceinline__ void normalise(uint8_t* to, int64_t pitch, const float* norm, const Job& j, int first, int stride, int B) {
  constexpr int NP = MAX_D / 128;
  const int lane = threadIdx.x & 31, K = j.K;
  const float inv = 1.0f / (float)K, eps = j.eps;
  uint2 in[NP];
  auto request = [&](int row) {
#pragma unroll
    for (int i = 0; i < NP; ++i)
      if (row < B && 4 * (lane + 32 * i) < K) in[i] = __ldcg(reinterpret_cast<const uint2*>(j.in + row * j.in_stride + 4 * (lane + 32 * i)));
  };
  request(first);
  for (int row = first; row < B; row += stride) {
    float f[NP][4];
    float sum = 0.0f;
#pragma unroll
    for (int i = 0; i < NP; ++i) {
      if (4 * (lane + 32 * i) < K) {
        const float2 a = unpack2(in[i].x), b = unpack2(in[i].y);
        f[i][0] = a.x; f[i][1] = a.y; f[i][2] = b.x; f[i][3] = b.y;
        sum += (a.x + a.y) + (b.x + b.y);
      }
    }
    request(row + stride);
    const float mean = warp_sum(sum) * inv;
    float sq = 0.0f;
#pragma unroll
    for (int i = 0; i < NP; ++i)
      if (4 * (lane + 32 * i) < K) {
#pragma unroll
        for (int k = 0; k < 4; ++k) { f[i][k] -= mean; sq += f[i][k] * f[i][k]; }
      }
    const float rstd = rsqrtf(warp_sum(sq) * inv + eps);
#pragma unroll
    for (int i = 0; i < NP; ++i) {
      const int c = 4 * (lane + 32 * i);
      if (c < K) {
        const float4 gw = *reinterpret_cast<const float4*>(norm + c), gb = *reinterpret_cast<const float4*>(norm + MAX_D + c);
        *reinterpret_cast<uint2*>(to + row * pitch + c * 2) = make_uint2(pack2(f[i][0] * rstd * gw.x + gb.x, f[i][1] * rstd * gw.y + gb.y),
                                                                         pack2(f[i][2] * rstd * gw.z + gb.z, f[i][3] * rstd * gw.w + gb.w));
      }
    }
  }
}

// The products of this CTA's weight rows, TPP tiles of eight at a time.  w holds the first pieces on entry.
template <int MT, int TPP, bool NORM>
__device__ __forceinline__ void project(uint8_t* sm, uint4 (&w)[PF], uint32_t bias, const Job& j, const Share& s, int B) {
  constexpr int STEPS = PF / TPP, RP = TPP * 8 + 2;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, pitch = norm_pitch(j.K);
  float* red = reinterpret_cast<float*>(sm + (NORM ? MT * 16 * pitch : 0));      // [WARPS][MT * 16][RP]
  // rows past the batch repeat its last row; their sums are dropped
  auto x_piece = [&](int row, int step) -> uint4 {
    row = min(row, B - 1);
    if constexpr (NORM) return *reinterpret_cast<const uint4*>(sm + row * pitch + (step * 32 + t * 8) * 2);
    else return ld_fresh(j.x + row * j.x_stride + step * 32 + t * 8);
  };
  constexpr int XB = MT == 1 ? (STEPS < 4 ? STEPS : 4) : MT == 2 ? (STEPS < 2 ? STEPS : 2) : 1;   // steps whose inputs are in flight together
  const int c_own = (threadIdx.x % (TPP * 4)) * 2;           // the column pair this thread finishes, in every row it takes
  for (int tile = s.c0; tile < s.c1; tile += TPP) {
    if (tile > s.c0) bias = fetch_bias<TPP>(j, s, tile);
    uint32_t res = 0;                                        // (written two phases ago or earlier)
    const int n_own = tile * 8 + c_own, row_own = threadIdx.x / (TPP * 4);
    if (j.residual && row_own < B && n_own < s.c1 * 8) res = __ldcg(reinterpret_cast<const unsigned*>(j.residual + row_own * j.res_stride + n_own));
    float acc[MT][TPP][4];
#pragma unroll
    for (int a = 0; a < MT; ++a)
#pragma unroll
      for (int c = 0; c < TPP; ++c)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[a][c][e] = 0.0f;
    for (int base = s.k0; base < s.k1; base += STEPS) {
      if (tile > s.c0 || base > s.k0) fetch_weights<TPP>(w, j, s, tile, base);
#pragma unroll
      for (int i0 = 0; i0 < STEPS; i0 += XB) {
        uint4 lo[XB][MT], hi[XB][MT];
#pragma unroll
        for (int i = 0; i < XB; ++i)
#pragma unroll
          for (int a = 0; a < MT; ++a) {
            const int step = min(base + i0 + i, s.k1 - 1);
            lo[i][a] = x_piece(a * 16 + g, step);
            hi[i][a] = x_piece(a * 16 + g + 8, step);
          }
#pragma unroll
        for (int i = 0; i < XB; ++i) {
          if (base + i0 + i >= s.k1) break;
#pragma unroll
          for (int a = 0; a < MT; ++a)
#pragma unroll
            for (int c = 0; c < TPP; ++c) {
              const uint4 b = w[(i0 + i) * TPP + c];         // (tiles past the CTA's share: stale, their sums are dropped)
              mma_16816(acc[a][c], lo[i][a].x, hi[i][a].x, lo[i][a].y, hi[i][a].y, b.x, b.y);
              mma_16816(acc[a][c], lo[i][a].z, hi[i][a].z, lo[i][a].w, hi[i][a].w, b.z, b.w);
            }
        }
      }
    }
#pragma unroll
    for (int a = 0; a < MT; ++a)
#pragma unroll
      for (int c = 0; c < TPP; ++c) {
        float* r = red + ((warp * MT + a) * 16 + g) * RP + c * 8 + 2 * t;
        *reinterpret_cast<float2*>(r) = make_float2(acc[a][c][0], acc[a][c][1]);
        *reinterpret_cast<float2*>(r + 8 * RP) = make_float2(acc[a][c][2], acc[a][c][3]);
      }
    __syncthreads();
    if (n_own < s.c1 * 8) {
      const float2 b = unpack2(bias);
      for (int row = row_own; row < B; row += THREADS / (TPP * 4)) {
        float2 v = make_float2(0.0f, 0.0f);
#pragma unroll
        for (int k = 0; k < WARPS; ++k) {
          const float2 f = *reinterpret_cast<const float2*>(red + (k * MT * 16 + row) * RP + c_own);
          v.x += f.x; v.y += f.y;
        }
        v.x = activate(j.act, v.x + b.x); v.y = activate(j.act, v.y + b.y);
        uint32_t out = pack2(v.x, v.y);
        if (j.residual) {
          if (row != row_own) res = __ldcg(reinterpret_cast<const unsigned*>(j.residual + row * j.res_stride + n_own));
          const float2 f = unpack2(out), r = unpack2(res);
          out = pack2(r.x + f.x, r.y + f.y);
        }
        *reinterpret_cast<uint32_t*>(j.y + row * j.y_stride + n_own) = out;
      }
    }
    __syncthreads();                              // (the sums are overwritten by the next tiles, or the next phase)
  }
}

// ---- phase 1: a group of 512, 256 or 128 threads takes (row, head) after (row, head) - as many groups as there are heads for
// an SM, one after another each costs 8000 cycles of latency; dv / 4 threads across the state's columns, PF passes of rows
// in flight
struct MixShape {
  int threads, group, tid, first, stride;         // of the group; its first (row, head) and the step to its next
  int ty_n, col, ty; bool live;
  __device__ __forceinline__ explicit MixShape(const TokenParams& p) {
    const int per_sm = (p.B * p.H + gridDim.x - 1) / gridDim.x, tx_n = p.dv >> 2;
    threads = per_sm <= 1 ? THREADS : per_sm == 2 ? THREADS / 2 : THREADS / 4;
    group = threadIdx.x / threads; tid = threadIdx.x % threads;
    first = blockIdx.x + group * gridDim.x; stride = gridDim.x * (THREADS / threads);
    ty_n = threads / tx_n; col = (tid % tx_n) * 4; ty = tid / tx_n; live = ty < ty_n;
  }
  __device__ __forceinline__ void sync() const { asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "r"(threads) : "memory"); }
};
__device__ __forceinline__ void fetch_state(uint4 (&r)[PF], const TokenParams& p, const fpb_decoder_layer& l, const MixShape& m, int unit, int row0) {
  const int64_t at = (unit / p.H) * l.prev_sb + (unit % p.H) * l.prev_sh + m.col;
#pragma unroll
  for (int u = 0; u < PF; ++u) {
    const int row = row0 + u * m.ty_n;
    r[u] = make_uint4(0u, 0u, 0u, 0u);
    if (!l.s_prev || !m.live || row >= p.dk || unit >= p.B * p.H) continue;
    if (p.prev_f32) r[u] = ld_stream((const float*)l.s_prev + at + (int64_t)row * p.dv);
    else {
      const uint2 v = __ldg(reinterpret_cast<const uint2*>((const bf16*)l.s_prev + at + (int64_t)row * p.dv));
      const float2 a = unpack2(v.x), b = unpack2(v.y);
      r[u] = make_uint4(__float_as_uint(a.x), __float_as_uint(a.y), __float_as_uint(b.x), __float_as_uint(b.y));
    }
  }
}
__device__ __forceinline__ void mix(float* sh, uint4 (&r)[PF], const TokenParams& p, const fpb_decoder_layer& l) {
  const MixShape m(p);
  float *sh_q = sh + m.group * 512, *sh_k = sh_q + 256, *sh_o = sh + 2048 + m.group * m.threads * 4;
  const int tid = m.tid, qk = p.H * p.dk, width = p.H * p.dv, pass = PF * m.ty_n;
  const float rs = rsqrtf((float)p.dk);
  for (int unit = m.first; unit < p.B * p.H; unit += m.stride) {
    const int b = unit / p.H, h = unit % p.H;
    const float gamma = p.gamma[h];
    const bf16* in = p.qkvg + (int64_t)b * (2 * qk + 2 * width);
    for (int i = tid; i < p.dk / 2; i += m.threads) {
      float2 q = unpack2(__ldcg(reinterpret_cast<const unsigned*>(in + h * p.dk + 2 * i)));
      float2 k = unpack2(__ldcg(reinterpret_cast<const unsigned*>(in + qk + h * p.dk + 2 * i)));
      if (l.phasors) {
        const float2 c = __ldg(reinterpret_cast<const float2*>(l.phasors) + i);
        q = make_float2(q.x * c.x - q.y * c.y, q.x * c.y + q.y * c.x);
        k = make_float2(k.x * c.x - k.y * c.y, k.x * c.y + k.y * c.x);
      }
      sh_q[2 * i] = q.x; sh_q[2 * i + 1] = q.y;
      sh_k[2 * i] = k.x * rs; sh_k[2 * i + 1] = k.y * rs;
    }
    float2 v01 = make_float2(0.f, 0.f), v23 = v01;
    if (m.live) {
      const uint2 v = __ldcg(reinterpret_cast<const uint2*>(in + 2 * qk + h * p.dv + m.col));
      v01 = unpack2(v.x); v23 = unpack2(v.y);
    }
    // GroupNorm and gate of the head: warp 0, channels 4 lane + 128 k
    float2 z[2][2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int c = 4 * tid + 128 * k;
      if (tid < 32 && c < p.dv) {
        const uint2 v = __ldcg(reinterpret_cast<const uint2*>(in + 2 * qk + width + h * p.dv + c));
        z[k][0] = unpack2(v.x); z[k][1] = unpack2(v.y);
      }
    }
    m.sync();
    float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
    const int64_t at = b * l.out_sb + h * l.out_sh + m.col;
    for (int r0 = m.ty; r0 < p.dk; r0 += pass) {
      if (r0 != m.ty) fetch_state(r, p, l, m, unit, r0);
#pragma unroll
      for (int u = 0; u < PF; ++u) {
        const int row = r0 + u * m.ty_n;
        if (!m.live || row >= p.dk) continue;
        const float kr = sh_k[row], qr = sh_q[row];
        float4 s;
        s.x = fmaf(gamma, __uint_as_float(r[u].x), kr * v01.x); s.y = fmaf(gamma, __uint_as_float(r[u].y), kr * v01.y);
        s.z = fmaf(gamma, __uint_as_float(r[u].z), kr * v23.x); s.w = fmaf(gamma, __uint_as_float(r[u].w), kr * v23.y);
        o.x = fmaf(qr, s.x, o.x); o.y = fmaf(qr, s.y, o.y); o.z = fmaf(qr, s.z, o.z); o.w = fmaf(qr, s.w, o.w);
        if (p.out_f32) *reinterpret_cast<float4*>((float*)l.s_out + at + (int64_t)row * p.dv) = s;
        else *reinterpret_cast<uint2*>((bf16*)l.s_out + at + (int64_t)row * p.dv) = make_uint2(pack2(s.x, s.y), pack2(s.z, s.w));
      }
    }
    if (unit + m.stride < p.B * p.H) fetch_state(r, p, l, m, unit + m.stride, m.ty);
    if (m.live) *reinterpret_cast<float4*>(sh_o + m.ty * p.dv + m.col) = o;
    m.sync();
    // (the other warps go on to the next head: its q and k have buffers of their own to wait for only at the barrier above)
    if (tid < 32) {
      float x[2][4];
      float sum = 0.0f;
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const int c = 4 * tid + 128 * k;
        x[k][0] = x[k][1] = x[k][2] = x[k][3] = 0.0f;
        if (c < p.dv)
          for (int y = 0; y < m.ty_n; ++y) {
            const float4 f = *reinterpret_cast<const float4*>(sh_o + y * p.dv + c);
            x[k][0] += f.x; x[k][1] += f.y; x[k][2] += f.z; x[k][3] += f.w;
          }
        sum += (x[k][0] + x[k][1]) + (x[k][2] + x[k][3]);
      }
      const float mean = warp_sum(sum) / (float)p.dv;
      float sq = 0.0f;
#pragma unroll
      for (int k = 0; k < 2; ++k)
        if (4 * tid + 128 * k < p.dv) {
#pragma unroll
          for (int e = 0; e < 4; ++e) { x[k][e] -= mean; sq += x[k][e] * x[k][e]; }
        }
      const float rstd = rsqrtf(warp_sum(sq) / (float)p.dv + (float)l.gn_eps);
      const int act = (int)l.act_gate;
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const int c = 4 * tid + 128 * k;
        if (c < p.dv)
          *reinterpret_cast<uint2*>(p.gated + (int64_t)b * width + h * p.dv + c) =
              make_uint2(pack2(x[k][0] * rstd * activate(act, z[k][0].x), x[k][1] * rstd * activate(act, z[k][0].y)),
                         pack2(x[k][2] * rstd * activate(act, z[k][1].x), x[k][3] * rstd * activate(act, z[k][1].y)));
      }
    }
  }
}

template <int MT, bool NORM>
__device__ __forceinline__ void project_any(uint8_t* sm, uint4 (&w)[PF], uint32_t bias, const Job& j, const Share& s, int B) {
  const int n = s.c1 - s.c0;
  if (n <= 1) project<MT, 1, NORM>(sm, w, bias, j, s, B);
  else if (n <= 2 || MT > 2) project<MT, 2, NORM>(sm, w, bias, j, s, B);
  else if constexpr (MT <= 2) project<MT, 4, NORM>(sm, w, bias, j, s, B);
}
template <int MT> __device__ __forceinline__ void prefetch(uint4 (&w)[PF], uint32_t& bias, const Job& j, const Share& s) {
  const int n = s.c1 - s.c0;
  if (n <= 1) { fetch_weights<1>(w, j, s, s.c0, s.k0); bias = fetch_bias<1>(j, s, s.c0); }
  else if (n <= 2 || MT > 2) { fetch_weights<2>(w, j, s, s.c0, s.k0); bias = fetch_bias<2>(j, s, s.c0); }
  else if constexpr (MT <= 2) { fetch_weights<4>(w, j, s, s.c0, s.k0); bias = fetch_bias<4>(j, s, s.c0); }
}

constexpr int NORM_BYTES = 2 * MAX_D * 4;         // staged norm parameters, ahead of the phases' own shared memory

// MT: batch rows / 16, rounded up
template <int MT>
__global__ void __launch_bounds__(THREADS, 1) token_kernel(const __grid_constant__ TokenParams p) {
  extern __shared__ __align__(16) uint8_t smem[];
  __shared__ int quit;
  __shared__ int2 tiles[5];                       // this CTA's share of each phase's weight rows / 8
  __shared__ Job jobs[2][5];                      // of this layer and the next ([1] is not used: no projection)
  float* norm = reinterpret_cast<float*>(smem);
  uint8_t* sm = smem + NORM_BYTES;
  uint4 w[PF];
  uint32_t bias = 0;
  unsigned passed = 0;
  if (threadIdx.x < 5) {
    const int width = p.H * p.dv, n = threadIdx.x == 0 ? 2 * p.H * p.dk + 2 * width : threadIdx.x == 3 ? p.ffn : width;
    const int64_t t = n >> 3, c = blockIdx.x, g = gridDim.x;
    tiles[threadIdx.x] = make_int2((int)(t * c / g), (int)(t * (c + 1) / g));
  }
  auto make_jobs = [&](int i) {                   // one warp, a phase a lane
    const int phase = threadIdx.x & 31;
    if (i < p.layers && phase < 5 && phase != 1) jobs[i & 1][phase] = job_of(p, i, phase, MT > 1);
  };
  if (threadIdx.x < 32) { make_jobs(0); make_jobs(1); }
  __syncthreads();
  // Into L2 two phases ahead, so that HBM streams all the time and the register prefetch at the end of a phase is short:
  // one bulk request a weight tile (eight rows) or state.
  auto request_l2 = [&](int i, int phase) {
    if (phase >= 5) { phase -= 5; ++i; }
    if (i >= p.layers || threadIdx.x >= 32) return;
    if (phase == 1) {
      const fpb_decoder_layer& l = p.layer[i];
      if (!l.s_prev) return;
      const int esize = p.prev_f32 ? 4 : 2, bytes = p.dk * p.dv * esize;
      for (int u = blockIdx.x + gridDim.x * threadIdx.x; u < p.B * p.H; u += gridDim.x * 32) {
        const char* at = (const char*)l.s_prev + ((u / p.H) * l.prev_sb + (u % p.H) * l.prev_sh) * esize;
        if (((uintptr_t)at | bytes) % 16 == 0) prefetch_l2(at, bytes);
      }
    } else {
      const Job& j = jobs[i & 1][phase];
      const int2 c = tiles[phase];
      for (int tile = c.x + threadIdx.x; tile < c.y; tile += 32) {
        const int m = matrix_of(j, tile * 8);
        prefetch_l2((const bf16*)j.w[m] + (int64_t)(tile * 8 - j.n_beg[m]) * j.K, 8 * j.K * 2);
      }
    }
  };
  auto ahead = [&](int i, int phase) {            // what the coming phase reads that no phase writes
    if (phase == 1) {
      const MixShape m(p);
      fetch_state(w, p, p.layer[i], m, m.first, m.ty);
      return;
    }
    const Job& j = jobs[i & 1][phase];
    prefetch<MT>(w, bias, j, share_of(j, tiles[phase]));
    if (phase == 0 || phase == 3) stage_norm(norm, j);
  };
  // Every CTA has arrived (what it wrote is visible), or the wait ran out: the CTA then reports it and leaves.  What the
  // next phases need besides the others' results is requested between the arrival and the wait.
  auto arrive = [&]() {
    ++passed;
    __syncthreads();
    if (threadIdx.x == 0) add_release(p.arrived);
  };
  auto wait = [&]() {
    if (threadIdx.x == 0) {
      const long long t0 = clock64();
      const unsigned want = passed * gridDim.x;
      int gone = 0;
      while (ld_acquire(p.arrived) < want)
        if (clock64() - t0 > p.wait_cycles) { gone = 1; break; }
      if (gone) atomicCAS(p.status, 0, 0x7f0);
      quit = gone;
    }
    copy_async_wait();
    __syncthreads();
    return quit == 0;
  };
  auto grid_meet = [&]() { arrive(); return wait(); };
  auto grid_sync = [&](int i, int phase) {        // ahead of that phase
    arrive();
    ahead(i, phase);
    request_l2(i, phase + 2);
    // the records of the layer after: their slot was last read by this layer's predecessor
    if (phase == 2 && (threadIdx.x >> 5) == WARPS - 1) make_jobs(i + 1);
    return wait();
  };
  ahead(0, 0);
  request_l2(0, 1);
  request_l2(0, 2);
  copy_async_wait();
  __syncthreads();
  for (int i = 0; i < p.layers; ++i) {
    for (int phase = 0; phase < 5; ++phase) {
      if (phase == 1) {
        mix(reinterpret_cast<float*>(sm), w, p, p.layer[i]);
      } else {
        const Job& j = jobs[i & 1][phase];
        const Share s = share_of(j, tiles[phase]);
        if (MT == 1 && (phase == 0 || phase == 3)) {
          normalise(sm, norm_pitch(j.K), norm, j, threadIdx.x >> 5, WARPS, p.B);
          __syncthreads();
          project_any<MT, MT == 1>(sm, w, bias, j, s, p.B);
        } else {
          if (MT > 1 && (phase == 0 || phase == 3)) {
            // warp 0 of the first B CTAs takes a row; everybody reads the result
            if (threadIdx.x < 32) normalise(reinterpret_cast<uint8_t*>(p.normed), j.K * 2, norm, j, blockIdx.x, gridDim.x, p.B);
            if (!grid_meet()) return;
          }
          project_any<MT, false>(sm, w, bias, j, s, p.B);
        }
      }
      if (i == p.layers - 1 && phase == 4) break;
      if (!(phase == 4 ? grid_sync(i + 1, 0) : grid_sync(i, phase + 1))) return;
    }
  }
}

template <int MT>
cudaError_t launch_token(const TokenParams& p, cudaStream_t stream) {
  constexpr int TPP = MT > 2 ? 2 : 4;
  constexpr int RED = WARPS * MT * 16 * (TPP * 8 + 2) * 4, MIX = (4 * 512 + THREADS * 4) * 4;
  constexpr int MOST = NORM_BYTES + (MT == 1 ? 16 * norm_pitch(MAX_D) : 0) + RED;
  static_assert(MOST <= 227 * 1024 && MIX <= RED, "shared memory of a CTA");
  static std::atomic<int> sms[64];
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  int n = dev >= 0 && dev < 64 ? sms[dev].load(std::memory_order_acquire) : 0;
  if (n == 0) {
    if ((e = cudaFuncSetAttribute(token_kernel<MT>, cudaFuncAttributeMaxDynamicSharedMemorySize, MOST)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
    if (dev >= 0 && dev < 64) sms[dev].store(n, std::memory_order_release);
  }
  if ((e = cudaMemsetAsync(p.arrived, 0, sizeof(unsigned), stream)) != cudaSuccess) return e;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(n); cfg.blockDim = dim3(THREADS); cfg.stream = stream;
  cfg.dynamicSmemBytes = NORM_BYTES + (MT == 1 ? 16 * norm_pitch(p.H * p.dv) : 0) + RED;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeCooperative;        // the CTAs wait for one another: all of them resident, or none starts
  attr.val.cooperative = 1;
  cfg.attrs = &attr; cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, token_kernel<MT>, p);
}

bool aligned(const void* p, int n) { return (uintptr_t)p % n == 0; }

}  // namespace

int64_t decoder_token_workspace(const fpb_token_dims& d) {
  const int64_t qk = (int64_t)d.H * d.dk, width = (int64_t)d.H * d.dv;
  return 2 * (int64_t)d.B * (2 * qk + 2 * width + 4 * width + d.ffn) + 256;    // TokenParams' buffers, bf16; barrier
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
    for (const float* v : {l.norm1_w, l.norm1_b, l.norm2_w, l.norm2_b})
      if (!aligned(v, 16)) return FPB_ERR_BAD_STRIDE;
    if (!aligned(l.phasors, 8)) return FPB_ERR_BAD_STRIDE;
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
  const int width = d.H * d.dv, qk = d.H * d.dk;
  TokenParams p;
  p.B = d.B; p.H = d.H; p.dk = d.dk; p.dv = d.dv; p.ffn = d.ffn;
  p.prev_f32 = d.prev_dtype == FPB_F32; p.out_f32 = d.out_dtype == FPB_F32;
  bf16* buf = (bf16*)d.workspace;
  p.arrived = (unsigned*)buf; buf += 64;
  auto take = [&](int64_t n) { bf16* r = buf; buf += n; return r; };       // (every row is a multiple of 16 bytes)
  p.qkvg = take((int64_t)d.B * (2 * qk + 2 * width));
  p.gated = take((int64_t)d.B * width);
  p.mid = take((int64_t)d.B * width);             // x + retention of the layer
  p.between = take((int64_t)d.B * width);         // x between layers
  p.hidden = take((int64_t)d.B * d.ffn);
  p.normed = take((int64_t)d.B * width);
  p.status = device_status_ptr();
  p.wait_cycles = walk_tuning().wait_cycles;
  if (!p.status) return FPB_ERR_LAUNCH;
  for (int h = 0; h < d.H; ++h) p.gamma[h] = gamma[h];
  for (int i0 = 0; i0 < d.layers; i0 += MAX_LAYERS) {
    const bool last = i0 + MAX_LAYERS >= d.layers;
    p.layers = last ? d.layers - i0 : MAX_LAYERS;
    // a launch after the first starts from the stream of x that the one before it ended in (`between` is next written by
    // the last phase of its first layer, long after everyone has read it)
    p.x = i0 == 0 ? (const bf16*)x : p.between; p.x_stride = i0 == 0 ? x_stride : width;
    p.y = last ? (bf16*)y : p.between; p.y_stride = last ? y_stride : width;
    for (int i = 0; i < p.layers; ++i) p.layer[i] = layers[i0 + i];
    const cudaError_t e = d.B <= 16 ? launch_token<1>(p, stream) : d.B <= 32 ? launch_token<2>(p, stream) : launch_token<4>(p, stream);
    if (e != cudaSuccess) return FPB_ERR_LAUNCH;
    ++*n_launched;
  }
  return FPB_OK;
}

}  // namespace fpb
