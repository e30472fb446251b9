// Chunked retention with fp32 arithmetic on the CUDA cores: forward and gradients of fp32 calls with head dimensions up
// to 128 (flash_pop/fused_retention/reference.py:10-111 is the same computation in PyTorch).
//
// The token-by-token walk (walk_generic.cu) is a serial chain of 0.45 us a token whatever the size: 4 launches of 117 us
// for B = 2, H = 4, T = 256, d = 64, 64 CTAs of 128 threads, nothing near saturated.  Chunks of 32 tokens turn the chain
// into small matrix products: per chunk (rs = 1/sqrt(dk), gamma^n from a table made in 64 bits)
//   forward   O_i  = sum_{j<=i} gamma^(i-j) (q_i . rs k_j) v_j + gamma^(i+1) q_i S          S  <- gamma^L S + sum_j gamma^(L-1-j) rs k_j (x) v_j
//   dQ        dQ_i = sum_{j<=i} gamma^(i-j) (dO_i . v_j) rs k_j + gamma^(i+1) S dO_i
//   dV        dV_j = rs sum_{i>=j} gamma^(i-j) (q_i . k_j) dO_i + gamma^(L-1-j) rs G^T k_j     G <- gamma^L G + sum_i gamma^(i+1) q_i (x) dO_i
//   dK        dK_j = rs sum_{i>=j} gamma^(i-j) (dO_i . v_j) q_i + gamma^(L-1-j) rs G v_j
// and T-segments of whole chunks fill the GPU: a pass over the segments' local end values, a scan over them, the walk
// proper with one CTA per (segment, head, row), dQ and dK/dV side by side in the backward.  The three launches are
// chained by programmatic dependent launch.  Every sum is made in runs of at most 32 products that are added up afterwards
// (as one chain of 128 the distance from 64 bits grew with the head dimension, 1.9e-7 -> 2.4e-7 at 128).
// Measured, token walk -> chunks, forward | backward: B=2 H=4 T=256 d=64 119 -> 14.5 | 354 -> 24.7 us; B=4 H=8 T=1024
// d=128 742 -> 193 | 2733 -> 450; B=64 H=16 T=256 d=64 552 -> 302 | 1657 -> 832.
//
// Bound by the FMA pipe and the shared-memory loads that feed it (16 FMAs per 16-byte load and thread at most); the chunk
// is as short as it is because the work inside a chunk grows with its length and the number of CTAs falls.
// Terms that the causal mask leaves out are never multiplied: an infinity in a later token must not reach an earlier one.
// Nor is padding - tokens past the end of a ragged chunk, channels past the head dimension: 0 x infinity would turn a
// token's own infinite gradient into NaN.
#include <atomic>

#include "fpb_common.cuh"

namespace fpb {
namespace {

constexpr int L32 = 32, THREADS = 256, PP = 36;        // tokens per chunk; pitch of a 32 x 32 score tile

struct ChunkParams {
  SeqView q, k, v, dO, o, dQ, dK, dV;
  StateView s0, s_out, g0, g_out;                       // start and end of the state walk; of the gradient's walk
  float *fwd, *rev;                                     // scratch (B, H, n_seg, dk, dv): start values of the segments
  int32_t T, H, B, dk, dv, n_seg, seg_len;
  int32_t n_fwd;                                        // z-blocks of the first role: state walk (B) or none (0)
  float gamma[FPB_MAX_HEADS];
};

__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// gamma^0 .. gamma^32, each product rounded once
__device__ __forceinline__ void power_table(float* pw, float gamma) {
  if (threadIdx.x <= L32) {
    double p = 1.0;
    for (int i = 0; i < (int)threadIdx.x; ++i) p *= (double)gamma;
    pw[threadIdx.x] = (float)p;
  }
}

// rows [t0, t0 + n) of a (T, D) tensor into a [32][W + 4] tile, zeros past n and past the d real columns
template <int W> __device__ __forceinline__ void load_tile(float* tile, const SeqView& s, int b, int h, int t0, int n, int d, float scale) {
  const float* src = (const float*)s.data + b * s.sb + h * s.sh;
  for (int i = threadIdx.x; i < L32 * W / 4; i += THREADS) {
    const int row = i / (W / 4), c = (i % (W / 4)) * 4;
    float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
    if (row < n && c < d) f = *reinterpret_cast<const float4*>(src + (int64_t)(t0 + row) * s.st + c);
    *reinterpret_cast<float4*>(tile + row * (W + 4) + c) = make_float4(f.x * scale, f.y * scale, f.z * scale, f.w * scale);
  }
}
template <int DK, int DV> __device__ __forceinline__ void load_state(float* S, const float* src, int dk, int dv) {
  for (int i = threadIdx.x; i < DK * DV / 4; i += THREADS) {
    const int row = i / (DV / 4), c = (i % (DV / 4)) * 4;
    float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
    if (src && row < dk && c < dv) f = *reinterpret_cast<const float4*>(src + row * dv + c);
    *reinterpret_cast<float4*>(S + row * (DV + 4) + c) = f;
  }
}
template <int DK, int DV> __device__ __forceinline__ void store_state(const float* S, float* dst, int dk, int dv) {
  for (int i = threadIdx.x; i < DK * DV / 4; i += THREADS) {
    const int row = i / (DV / 4), c = (i % (DV / 4)) * 4;
    if (row < dk && c < dv) *reinterpret_cast<float4*>(dst + row * dv + c) = *reinterpret_cast<const float4*>(S + row * (DV + 4) + c);
  }
}

// S <- decay S + sum over the chunk's n tokens of w_j A_j (x) B_j, w_j = pw[first + step * j]; a thread holds a
// (DK/16) x (DV/16) block of S, rows side by side, columns in pieces of four.  Padding of S - rows from dk, columns from dv
// on, none where EXACT - stays the zero it was loaded as.
template <int DK, int DV, bool EXACT> __device__ __forceinline__ void update_state(float* S, const float* A, const float* B, const float* pw, int n,
                                                                       int first, int step, float decay, int dk, int dv) {
  constexpr int TR = DK / 16, TC = DV / 16, CV = TC < 4 ? TC : 4, NC = TC / CV;
  const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;
  float acc[TR][TC];
  float* s0 = S + ty * TR * (DV + 4) + tx * CV;
#pragma unroll
  for (int r = 0; r < TR; ++r)
#pragma unroll
    for (int c = 0; c < TC; ++c) acc[r][c] = 0.0f;
#pragma unroll 2
  for (int j = 0; j < n; ++j) {
    const float w = pw[first + step * j];
    float a[TR], b[TC];
    const float* ar = A + j * (DK + 4) + ty * TR;
    const float* br = B + j * (DV + 4) + tx * CV;
#pragma unroll
    for (int r = 0; r < TR; ++r) a[r] = w * ar[r];
#pragma unroll
    for (int c = 0; c < TC; ++c) b[c] = br[(c / CV) * (DV / NC) + c % CV];
#pragma unroll
    for (int r = 0; r < TR; ++r)
#pragma unroll
      for (int c = 0; c < TC; ++c) acc[r][c] = fmaf(a[r], b[c], acc[r][c]);
  }
#pragma unroll
  for (int r = 0; r < TR; ++r)
#pragma unroll
    for (int c = 0; c < TC; ++c) {
      const int col = (c / CV) * (DV / NC) + c % CV;
      float& x = s0[r * (DV + 4) + col];
      if (EXACT || (ty * TR + r < dk && tx * CV + col < dv)) x = fmaf(decay, x, acc[r][c]);
    }
}

__device__ __forceinline__ float dot4(float4 a, float4 b, float c) {
  return fmaf(a.x, b.x, fmaf(a.y, b.y, fmaf(a.z, b.z, fmaf(a.w, b.w, c))));
}
// P[x][y] = gamma^|x-y| (X_x . Y_y) on the causal side (y <= x, or y >= x with UP): eight threads a row, four y's each
template <int W, bool UP> __device__ __forceinline__ void scores(float* P, const float* X, const float* Y, const float* pw) {
  const int x = threadIdx.x >> 3, y0 = threadIdx.x & 7;
  float acc[4] = {0.f, 0.f, 0.f, 0.f};
  const float* xr = X + x * (W + 4);
  for (int k0 = 0; k0 < W; k0 += 32) {
    float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
    for (int k = k0; k < k0 + 32; k += 4) {
      const float4 a = *reinterpret_cast<const float4*>(xr + k);
#pragma unroll
      for (int m = 0; m < 4; ++m) sum[m] = dot4(a, *reinterpret_cast<const float4*>(Y + (y0 + 8 * m) * (W + 4) + k), sum[m]);
    }
#pragma unroll
    for (int m = 0; m < 4; ++m) acc[m] += sum[m];
  }
#pragma unroll
  for (int m = 0; m < 4; ++m) {
    const int y = y0 + 8 * m, gap = UP ? y - x : x - y;
    P[x * PP + y] = gap >= 0 ? acc[m] * pw[gap] : 0.0f;
  }
}

// The thread's rows and columns of a [32][W] output tile: W/32 rows side by side, four columns - side by side (STRIDED
// false, one 16-byte access) or W/4 apart (STRIDED true: the columns of a product with the transposed state).
template <int W> struct Own {
  static constexpr int ROWS = W / 32, GROUPS = W / 4;
  int row, col;
  __device__ __forceinline__ Own(bool strided) : row((threadIdx.x / GROUPS) * ROWS), col((threadIdx.x % GROUPS) * (strided ? 1 : 4)) {}
};
template <int R> __device__ __forceinline__ void add_to(float (&acc)[R][4], const float (&sum)[R][4]) {
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[r][c] += sum[r][c];
}
// acc += A[row] M  for the [K][N] matrix M (pitch N + 4)
template <int K, int N> __device__ __forceinline__ void times(float (&acc)[N / 32][4], const float* A, const float* M, const Own<N>& own) {
  for (int k0 = 0; k0 < K; k0 += 32) {
    float sum[N / 32][4] = {};
#pragma unroll 2
    for (int k = k0; k < k0 + 32; k += 4) {
      float4 m[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) m[i] = *reinterpret_cast<const float4*>(M + (k + i) * (N + 4) + own.col);
#pragma unroll
      for (int r = 0; r < N / 32; ++r) {
        const float4 a = *reinterpret_cast<const float4*>(A + (own.row + r) * (K + 4) + k);
        const float e[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          sum[r][0] = fmaf(e[i], m[i].x, sum[r][0]); sum[r][1] = fmaf(e[i], m[i].y, sum[r][1]);
          sum[r][2] = fmaf(e[i], m[i].z, sum[r][2]); sum[r][3] = fmaf(e[i], m[i].w, sum[r][3]);
        }
      }
    }
    add_to<N / 32>(acc, sum);
  }
}
// acc += A[row] M^T for the [N][K] matrix M (pitch K + 4), columns N/4 apart
template <int K, int N> __device__ __forceinline__ void times_t(float (&acc)[N / 32][4], const float* A, const float* M, const Own<N>& own) {
  for (int k0 = 0; k0 < K; k0 += 32) {
    float sum[N / 32][4] = {};
#pragma unroll 2
    for (int k = k0; k < k0 + 32; k += 4) {
      float4 m[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) m[i] = *reinterpret_cast<const float4*>(M + (own.col + i * (N / 4)) * (K + 4) + k);
#pragma unroll
      for (int r = 0; r < N / 32; ++r) {
        const float4 a = *reinterpret_cast<const float4*>(A + (own.row + r) * (K + 4) + k);
#pragma unroll
        for (int i = 0; i < 4; ++i) sum[r][i] = dot4(a, m[i], sum[r][i]);
      }
    }
    add_to<N / 32>(acc, sum);
  }
}
// acc += P[row] M over the causal side of the 32 x 32 tile P (y <= row, or row <= y < n with UP), M [32][N]
template <int N, bool STRIDED, bool UP> __device__ __forceinline__ void times_scores(float (&acc)[N / 32][4], const float* P, const float* M,
                                                                                    const Own<N>& own, int n) {
  constexpr int R = N / 32;
  float sum[R][4] = {};
  const int lo = UP ? own.row & ~3 : 0, hi = UP ? n & ~3 : (own.row + R + 3) & ~3;
  for (int k = lo; k < hi; k += 4) {
    const bool whole = UP ? k >= own.row + R - 1 : k + 3 <= own.row;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float4 m;
      const float* mr = M + (k + i) * (N + 4) + own.col;
      if (STRIDED) m = make_float4(mr[0], mr[N / 4], mr[N / 2], mr[3 * N / 4]);
      else m = *reinterpret_cast<const float4*>(mr);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int row = own.row + r;
        if (whole || (UP ? k + i >= row : k + i <= row)) {
          const float e = P[row * PP + k + i];
          sum[r][0] = fmaf(e, m.x, sum[r][0]); sum[r][1] = fmaf(e, m.y, sum[r][1]);
          sum[r][2] = fmaf(e, m.z, sum[r][2]); sum[r][3] = fmaf(e, m.w, sum[r][3]);
        }
      }
    }
  }
  if (UP) {                                        // the last, broken group of four of a ragged chunk
    for (int k = max(hi, lo); k < n; ++k) {
      const float* mr = M + k * (N + 4) + own.col;
#pragma unroll
      for (int r = 0; r < R; ++r) {
        if (k < own.row + r) continue;
        const float e = P[(own.row + r) * PP + k];
#pragma unroll
        for (int c = 0; c < 4; ++c) sum[r][c] = fmaf(e, mr[STRIDED ? c * (N / 4) : c], sum[r][c]);
      }
    }
  }
  add_to<R>(acc, sum);
}
template <int N> __device__ __forceinline__ void scale_rows(float (&acc)[N / 32][4], const Own<N>& own, const float* pw, int first, int step, int n) {
#pragma unroll
  for (int r = 0; r < N / 32; ++r) {
    const float z = own.row + r < n ? pw[first + step * (own.row + r)] : 0.0f;
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[r][c] *= z;
  }
}
template <int N, bool STRIDED> __device__ __forceinline__ void store_rows(const float (&acc)[N / 32][4], const Own<N>& own, const SeqView& s, int b,
                                                                         int h, int t0, int n, int d, float scale) {
  float* dst = (float*)s.data + b * s.sb + h * s.sh;
#pragma unroll
  for (int r = 0; r < N / 32; ++r) {
    if (own.row + r >= n) continue;
    float* p = dst + (int64_t)(t0 + own.row + r) * s.st;
    if constexpr (STRIDED) {
#pragma unroll
      for (int c = 0; c < 4; ++c)
        if (own.col + c * (N / 4) < d) p[own.col + c * (N / 4)] = acc[r][c] * scale;
    } else if (own.col < d) {
      *reinterpret_cast<float4*>(p + own.col) = make_float4(acc[r][0] * scale, acc[r][1] * scale, acc[r][2] * scale, acc[r][3] * scale);
    }
  }
}

template <int DK, int DV> struct Smem {
  static constexpr int S = DK * (DV + 4), TK = L32 * (DK + 4), TV = L32 * (DV + 4), P = L32 * PP, PW = 36;
  static constexpr int TILES2 = (S + TK + TV + PW) * 4, FWD = (S + 2 * TK + TV + P + PW) * 4, BWD = (S + 2 * TK + 2 * TV + 2 * P + PW) * 4;
};

__device__ __forceinline__ float* slot_of(float* base, const ChunkParams& p, int b, int h, int seg) {
  return base + (((int64_t)b * p.H + h) * p.n_seg + seg) * p.dk * p.dv;
}

// Local end values of the segments, from zero: grid (n_seg - 1, H, roles * B).  Role 0: the state over (k, v), every
// segment but the last; role 1: its gradient over (q, dO), every segment but the first.
template <int DK, int DV, bool EXACT>
__global__ void __launch_bounds__(THREADS) chunk_segments_kernel(const __grid_constant__ ChunkParams p) {
  using M = Smem<DK, DV>;
  extern __shared__ __align__(16) float sm[];
  float *S = sm, *A = S + M::S, *B = A + M::TK, *pw = B + M::TV;
  const bool rev = (int)blockIdx.z >= p.n_fwd;
  const int b = rev ? blockIdx.z - p.n_fwd : blockIdx.z, h = blockIdx.y, seg = blockIdx.x + (rev ? 1 : 0);
  const int t0 = seg * p.seg_len, t1 = min(t0 + p.seg_len, p.T), chunks = (t1 - t0 + L32 - 1) / L32;
  power_table(pw, p.gamma[h]);
  load_state<DK, DV>(S, nullptr, p.dk, p.dv);
  const float rs = 1.0f / sqrtf((float)p.dk);
  for (int c = 0; c < chunks; ++c) {
    const int a = t0 + (rev ? chunks - 1 - c : c) * L32, n = min(L32, t1 - a);
    load_tile<DK>(A, rev ? p.q : p.k, b, h, a, n, p.dk, rev ? 1.0f : rs);
    load_tile<DV>(B, rev ? p.dO : p.v, b, h, a, n, p.dv, 1.0f);
    __syncthreads();
    update_state<DK, DV, EXACT>(S, A, B, pw, n, rev ? 1 : n - 1, rev ? 1 : -1, pw[n], p.dk, p.dv);
    __syncthreads();
  }
  grid_wait();                                     // (the first of the chain: nothing to wait for)
  grid_release();
  store_state<DK, DV>(S, slot_of(rev ? p.rev : p.fwd, p, b, h, seg), p.dk, p.dv);
}

// The scan: slot s <- start value of segment s.  One thread carries four state elements, eight local values ahead of
// the running one (they do not depend on it).  grid (dk dv / 1024, H, roles * B)
__global__ void __launch_bounds__(THREADS) chunk_scan_kernel(const __grid_constant__ ChunkParams p) {
  grid_wait();
  grid_release();
  const bool rev = (int)blockIdx.z >= p.n_fwd;
  const int b = rev ? blockIdx.z - p.n_fwd : blockIdx.z, h = blockIdx.y, e = (blockIdx.x * THREADS + threadIdx.x) * 4, size = p.dk * p.dv;
  if (e >= size) return;
  const StateView& from = rev ? p.g0 : p.s0;
  float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
  if (from.data) a = *reinterpret_cast<const float4*>((const float*)from.data + b * from.sb + h * from.sh + e);
  float* base = slot_of(rev ? p.rev : p.fwd, p, b, h, 0) + e;
  const double g = (double)p.gamma[h];
  auto power = [&](int n) { double r = 1.0, f = g; for (; n; n >>= 1, f *= f) if (n & 1) r *= f; return (float)r; };
  const float whole = power(p.seg_len), tail = power(p.T - (p.n_seg - 1) * p.seg_len);
  constexpr int AHEAD = 8;
  for (int i0 = 0; i0 < p.n_seg; i0 += AHEAD) {
    float4 loc[AHEAD];
#pragma unroll
    for (int i = 0; i < AHEAD; ++i) {
      const int s = rev ? p.n_seg - 1 - i0 - i : i0 + i;
      if (i0 + i < p.n_seg - 1) loc[i] = *reinterpret_cast<const float4*>(base + (int64_t)s * size);
    }
#pragma unroll
    for (int i = 0; i < AHEAD; ++i) {
      const int s = rev ? p.n_seg - 1 - i0 - i : i0 + i;
      if (i0 + i < p.n_seg) *reinterpret_cast<float4*>(base + (int64_t)s * size) = a;
      if (i0 + i < p.n_seg - 1) {
        const float f = s == p.n_seg - 1 ? tail : whole;
        a.x = fmaf(f, a.x, loc[i].x); a.y = fmaf(f, a.y, loc[i].y); a.z = fmaf(f, a.z, loc[i].z); a.w = fmaf(f, a.w, loc[i].w);
      }
    }
  }
}

// where a segment's walk starts
__device__ __forceinline__ const float* start_of(const ChunkParams& p, float* scratch, const StateView& s, int b, int h, int seg) {
  if (p.n_seg > 1) return slot_of(scratch, p, b, h, seg);
  return s.data ? (const float*)s.data + b * s.sb + h * s.sh : nullptr;
}

template <int DK, int DV, bool EXACT>
__global__ void __launch_bounds__(THREADS) chunk_fwd_kernel(const __grid_constant__ ChunkParams p) {
  using M = Smem<DK, DV>;
  extern __shared__ __align__(16) float sm[];
  float *S = sm, *Q = S + M::S, *K = Q + M::TK, *V = K + M::TK, *P = V + M::TV, *pw = P + M::P;
  const int b = blockIdx.z, h = blockIdx.y, seg = blockIdx.x, t0 = seg * p.seg_len, t1 = min(t0 + p.seg_len, p.T);
  const bool ends = seg == p.n_seg - 1 && p.s_out.data;
  const float rs = 1.0f / sqrtf((float)p.dk);
  power_table(pw, p.gamma[h]);
  const Own<DV> own(false);
  for (int a = t0; a < t1; a += L32) {
    const int n = min(L32, t1 - a);
    load_tile<DK>(Q, p.q, b, h, a, n, p.dk, 1.0f);
    load_tile<DK>(K, p.k, b, h, a, n, p.dk, rs);
    load_tile<DV>(V, p.v, b, h, a, n, p.dv, 1.0f);
    if (a == t0) {
      grid_wait();                                 // the segments' start values
      grid_release();
      load_state<DK, DV>(S, start_of(p, p.fwd, p.s0, b, h, seg), p.dk, p.dv);
    }
    __syncthreads();
    scores<DK, false>(P, Q, K, pw);
    float acc[DV / 32][4] = {};
    times<DK, DV>(acc, Q, S, own);
    scale_rows<DV>(acc, own, pw, 1, 1, n);
    __syncthreads();
    times_scores<DV, false, false>(acc, P, V, own, n);
    store_rows<DV, false>(acc, own, p.o, b, h, a, n, p.dv, 1.0f);
    if (a + L32 < t1 || ends) update_state<DK, DV, EXACT>(S, K, V, pw, n, n - 1, -1, pw[n], p.dk, p.dv);   // (S was last read before the barrier)
    __syncthreads();
  }
  if (ends) store_state<DK, DV>(S, (float*)p.s_out.data + b * p.s_out.sb + h * p.s_out.sh, p.dk, p.dv);
}

// z-blocks below n_fwd: dQ (forward walk over the state); the others: dK, dV, dS_0 (reverse walk over its gradient)
template <int DK, int DV, bool EXACT>
__global__ void __launch_bounds__(THREADS) chunk_bwd_kernel(const __grid_constant__ ChunkParams p) {
  using M = Smem<DK, DV>;
  extern __shared__ __align__(16) float sm[];
  float *S = sm, *Q = S + M::S, *K = Q + M::TK, *V = K + M::TK, *D = V + M::TV, *P1 = D + M::TV, *P2 = P1 + M::P, *pw = P2 + M::P;
  const bool rev = (int)blockIdx.z >= p.n_fwd;
  const int b = rev ? blockIdx.z - p.n_fwd : blockIdx.z, h = blockIdx.y, seg = blockIdx.x;
  const int t0 = seg * p.seg_len, t1 = min(t0 + p.seg_len, p.T), chunks = (t1 - t0 + L32 - 1) / L32;
  const float rs = 1.0f / sqrtf((float)p.dk);
  power_table(pw, p.gamma[h]);
  const Own<DK> own_k(true);
  const Own<DV> own_v(false);
  for (int c = 0; c < chunks; ++c) {
    const int a = t0 + (rev ? chunks - 1 - c : c) * L32, n = min(L32, t1 - a);
    if (rev) load_tile<DK>(Q, p.q, b, h, a, n, p.dk, 1.0f);
    load_tile<DK>(K, p.k, b, h, a, n, p.dk, rs);
    load_tile<DV>(V, p.v, b, h, a, n, p.dv, 1.0f);
    load_tile<DV>(D, p.dO, b, h, a, n, p.dv, 1.0f);
    if (c == 0) {
      grid_wait();
      grid_release();
      load_state<DK, DV>(S, rev ? start_of(p, p.rev, p.g0, b, h, seg) : start_of(p, p.fwd, p.s0, b, h, seg), p.dk, p.dv);
    }
    __syncthreads();
    if (!rev) {
      scores<DV, false>(P2, D, V, pw);
      float acc[DK / 32][4] = {};
      times_t<DV, DK>(acc, D, S, own_k);
      scale_rows<DK>(acc, own_k, pw, 1, 1, n);
      __syncthreads();
      times_scores<DK, true, false>(acc, P2, K, own_k, n);
      store_rows<DK, true>(acc, own_k, p.dQ, b, h, a, n, p.dk, 1.0f);
      if (c + 1 < chunks) update_state<DK, DV, EXACT>(S, K, V, pw, n, n - 1, -1, pw[n], p.dk, p.dv);
    } else {
      scores<DK, true>(P1, K, Q, pw);              // (K carries rs)
      scores<DV, true>(P2, V, D, pw);
      float av[DV / 32][4] = {};
      times<DK, DV>(av, K, S, own_v);
      scale_rows<DV>(av, own_v, pw, n - 1, -1, n);
      float ak[DK / 32][4] = {};
      times_t<DV, DK>(ak, V, S, own_k);
      scale_rows<DK>(ak, own_k, pw, n - 1, -1, n);
      __syncthreads();
      times_scores<DV, false, true>(av, P1, D, own_v, n);
      store_rows<DV, false>(av, own_v, p.dV, b, h, a, n, p.dv, 1.0f);
      times_scores<DK, true, true>(ak, P2, Q, own_k, n);
      store_rows<DK, true>(ak, own_k, p.dK, b, h, a, n, p.dk, rs);
      if (c + 1 < chunks || (seg == 0 && p.g_out.data)) update_state<DK, DV, EXACT>(S, Q, D, pw, n, 1, 1, pw[n], p.dk, p.dv);
    }
    __syncthreads();
  }
  if (rev && seg == 0 && p.g_out.data) store_state<DK, DV>(S, (float*)p.g_out.data + b * p.g_out.sb + h * p.g_out.sh, p.dk, p.dv);
}

cudaError_t launch(void (*kernel)(ChunkParams), dim3 grid, size_t smem, bool chained, const ChunkParams& p, cudaStream_t stream) {
  return launch_kernel(kernel, grid, THREADS, smem, chained, p, stream);
}

enum Pass { SEGMENTS, FORWARD, BACKWARD };
template <int DK, int DV, bool EXACT>
cudaError_t launch_pass_t(Pass pass, dim3 grid, bool chained, const ChunkParams& p, cudaStream_t stream) {
  using M = Smem<DK, DV>;
  static_assert(M::BWD <= 227 * 1024, "shared memory of a CTA");
  static std::atomic<bool> configured[64];
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64 || !configured[dev].load(std::memory_order_acquire)) {
    cudaError_t e;
    if ((e = cudaFuncSetAttribute(chunk_segments_kernel<DK, DV, EXACT>, cudaFuncAttributeMaxDynamicSharedMemorySize, M::TILES2)) != cudaSuccess) return e;
    if ((e = cudaFuncSetAttribute(chunk_fwd_kernel<DK, DV, EXACT>, cudaFuncAttributeMaxDynamicSharedMemorySize, M::FWD)) != cudaSuccess) return e;
    if ((e = cudaFuncSetAttribute(chunk_bwd_kernel<DK, DV, EXACT>, cudaFuncAttributeMaxDynamicSharedMemorySize, M::BWD)) != cudaSuccess) return e;
    if (dev >= 0 && dev < 64) configured[dev].store(true, std::memory_order_release);
  }
  if (pass == SEGMENTS) return launch(chunk_segments_kernel<DK, DV, EXACT>, grid, M::TILES2, chained, p, stream);
  if (pass == FORWARD) return launch(chunk_fwd_kernel<DK, DV, EXACT>, grid, M::FWD, chained, p, stream);
  return launch(chunk_bwd_kernel<DK, DV, EXACT>, grid, M::BWD, chained, p, stream);
}
cudaError_t launch_pass(Pass pass, dim3 grid, bool chained, const ChunkParams& p, cudaStream_t stream) {
  auto tile = [](int d) { return d <= 32 ? 32 : d <= 64 ? 64 : 128; };
  const int key = tile(p.dk) * 1000 + tile(p.dv);
  const bool exact = tile(p.dk) == p.dk && tile(p.dv) == p.dv;
  switch (key) {
#define FPB_CHUNK_CASE(DK_, DV_) case DK_ * 1000 + DV_: \
    return exact ? launch_pass_t<DK_, DV_, true>(pass, grid, chained, p, stream) : launch_pass_t<DK_, DV_, false>(pass, grid, chained, p, stream)
    FPB_CHUNK_CASE(32, 32); FPB_CHUNK_CASE(32, 64); FPB_CHUNK_CASE(32, 128);
    FPB_CHUNK_CASE(64, 32); FPB_CHUNK_CASE(64, 64); FPB_CHUNK_CASE(64, 128);
    FPB_CHUNK_CASE(128, 32); FPB_CHUNK_CASE(128, 64); FPB_CHUNK_CASE(128, 128);
#undef FPB_CHUNK_CASE
  }
  return cudaErrorInvalidValue;
}

// Segments of whole chunks: as many as the CTAs that fit the GPU at once (one an SM at 128 wide, two below), each at
// least one chunk; no more than the scratch holds; none where they do not pay.  In tenths of a chunk a sequence costs 10 a
// chunk whole, in segments 16 a chunk of one (state pass and walk) and 30 where they fill the GPU.  Measured, forward | backward
// in us, whole against split: 64 heads, d = 64, T = 33 14.7 | 20.1 against 23.6 | 31.0 (the token walk 18.3 | 51.3), T = 160
// 36.4 | 55.6 against 45.1 | 62.3, T = 300 70.0 | 107 against 69.8 | 104, T = 1024 223 | 405 against 184 | 303; 8 heads, T = 96
// 21.8 | 33.7 against 14.0 | 18.5; 64 heads, d = 128, T = 300 140 | 233 against 114 | 258, T = 1024 570 | 873 against 431 | 879.
void choose(ChunkParams& p, int64_t scratch_bytes, int directions) {
  const int chunks = (p.T + L32 - 1) / L32;
  const int64_t units = (int64_t)p.B * p.H, slots = (int64_t)sm_count() * ((p.dk > 64 && p.dv > 64) ? 1 : 2);
  int64_t n = units > 0 ? slots / units : 1;
  if (scratch_bytes >= 0) {
    const int64_t fit = scratch_bytes / (units * p.dk * p.dv * 4 * directions);
    n = n < fit ? n : fit;
  }
  n = n < chunks ? n : chunks;
  p.n_seg = 1; p.seg_len = chunks * L32;
  if (n < 2) return;
  const int per = (int)((chunks + n - 1) / n), count = (chunks + per - 1) / per;
  if (16 * per + 30 * units * count / slots >= 10 * chunks) return;
  p.seg_len = per * L32;
  p.n_seg = count;
}

bool seq_ok(const SeqView& s, int B, int T, int H) {
  return s.data && (uintptr_t)s.data % 16 == 0 && (B <= 1 || s.sb % 4 == 0) && (T <= 1 || s.st % 4 == 0) && (H <= 1 || s.sh % 4 == 0);
}
bool state_ok(const StateView& s, int B, int H) {
  return !s.data || ((uintptr_t)s.data % 16 == 0 && (B <= 1 || s.sb % 4 == 0) && (H <= 1 || s.sh % 4 == 0));
}
// Shorter sequences stay with the token walk: a chunk costs what a dozen of its tokens do, whatever it holds (forward at
// d = 64: 8.4 us a chunk, the walk 6.3 us at T = 8, 8.3 at 12, 10.4 at 16; at 128 x 128 13.9 us against 14.5 at T = 16).
constexpr int kMinTokens = 16;

bool common_ok(const ChunkArgs& a) {
  return a.T >= kMinTokens && a.dk <= 128 && a.dv <= 128 && a.dk % 4 == 0 && a.dv % 4 == 0 && a.B <= 32767 && a.H <= 65535 &&
         seq_ok(a.q, a.B, a.T, a.H) && seq_ok(a.k, a.B, a.T, a.H) && seq_ok(a.v, a.B, a.T, a.H) && state_ok(a.s0, a.B, a.H);
}
void fill(ChunkParams& p, const ChunkArgs& a) {
  p = ChunkParams{};
  p.q = a.q; p.k = a.k; p.v = a.v; p.dO = a.dO; p.o = a.o; p.dQ = a.dQ; p.dK = a.dK; p.dV = a.dV;
  p.s0 = a.s0; p.s_out = a.s_out; p.g0 = a.d_s_out; p.g_out = a.d_s0;
  p.T = a.T; p.H = a.H; p.B = a.B; p.dk = a.dk; p.dv = a.dv;
  for (int h = 0; h < a.H; ++h) p.gamma[h] = a.gamma[h];
}
int run(ChunkParams& p, Pass pass, int roles, cudaStream_t stream, int* n_launched) {
  cudaError_t e = cudaSuccess;
  const bool split = p.n_seg > 1;
  if (split) {
    if ((e = launch_pass(SEGMENTS, dim3(p.n_seg - 1, p.H, roles * p.B), false, p, stream)) != cudaSuccess) return FPB_ERR_LAUNCH;
    if ((e = launch(chunk_scan_kernel, dim3((p.dk * p.dv + THREADS * 4 - 1) / (THREADS * 4), p.H, roles * p.B), 0, true, p, stream)) != cudaSuccess)
      return FPB_ERR_LAUNCH;
    *n_launched += 2;
  }
  if ((e = launch_pass(pass, dim3(p.n_seg, p.H, roles * p.B), split, p, stream)) != cudaSuccess) return FPB_ERR_LAUNCH;
  ++*n_launched;
  return FPB_OK;
}

}  // namespace

int64_t chunk_f32_workspace(int B, int T, int H, int dk, int dv) {
  if (T < kMinTokens || dk > 128 || dv > 128 || dk % 4 || dv % 4) return 0;
  ChunkParams p{};
  p.B = B; p.T = T; p.H = H; p.dk = dk; p.dv = dv;
  choose(p, -1, 2);
  return p.n_seg > 1 ? (int64_t)B * H * p.n_seg * dk * dv * 4 * 2 : 0;      // the backward scans the state and its gradient
}

int launch_chunk_fwd(const ChunkArgs& a, cudaStream_t stream, int* n_launched) {
  if (!common_ok(a) || !seq_ok(a.o, a.B, a.T, a.H) || !state_ok(a.s_out, a.B, a.H)) return FPB_CHUNK_NOT_APPLICABLE;
  ChunkParams p;
  fill(p, a);
  p.n_fwd = a.B;
  choose(p, a.scratch ? a.scratch_bytes : 0, 1);
  p.fwd = a.scratch;
  return run(p, FORWARD, 1, stream, n_launched);
}

int launch_chunk_bwd(const ChunkArgs& a, bool skip_dq, bool skip_dkdv, cudaStream_t stream, int* n_launched) {
  if (!common_ok(a) || !seq_ok(a.dO, a.B, a.T, a.H) || !state_ok(a.d_s_out, a.B, a.H) || !state_ok(a.d_s0, a.B, a.H)) return FPB_CHUNK_NOT_APPLICABLE;
  if ((!skip_dq && !seq_ok(a.dQ, a.B, a.T, a.H)) || (!skip_dkdv && (!seq_ok(a.dK, a.B, a.T, a.H) || !seq_ok(a.dV, a.B, a.T, a.H))))
    return FPB_CHUNK_NOT_APPLICABLE;
  if (skip_dq && skip_dkdv) return FPB_OK;
  ChunkParams p;
  fill(p, a);
  const int roles = (skip_dq ? 0 : 1) + (skip_dkdv ? 0 : 1);
  p.n_fwd = skip_dq ? 0 : a.B;
  choose(p, a.scratch ? a.scratch_bytes : 0, roles);
  p.fwd = a.scratch;
  p.rev = a.scratch ? a.scratch + (skip_dq ? 0 : (int64_t)a.B * a.H * p.n_seg * a.dk * a.dv) : nullptr;
  return run(p, BACKWARD, roles, stream, n_launched);
}

}  // namespace fpb
