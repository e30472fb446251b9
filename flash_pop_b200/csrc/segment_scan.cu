// T-segments for under-filled launches of the retention walks.
//
// A walk is one CTA per (batch, head, state tile), strictly sequential over the T/64 chunks of its sequence, so a
// call with few sequences leaves most of the GPU idle (the reference's grid has the same shape:
// flash_pop/fused_retention/fused_chunk_fwd.py:119).  The retention recurrence is linear in the state,
//     S_end = gamma^len S_start + E,   E = the end value of the same piece walked from a zero state,
// so a sequence can be cut into n pieces that are walked concurrently:
//   1. every piece but the last computes its local end value E_s from a zero start (state-only instance of the scan
//      kernel: it reads the two operands of the increment and nothing else) into fp32 scratch memory (B, H, n, dk, dv);
//   2. this file's kernel scans the pieces of each (batch, head): A_0 = S_0, A_{s+1} = gamma^len_s A_s + E_s, and
//      writes A_s over E_s;
//   3. the walk proper runs one CTA per piece from A_s; the last piece ends in the call's end state.
// Reverse walks (the state gradient) are the mirror image: pieces are scanned from the last to the first.
// Everything is deterministic; results differ from the unsplit walk by fp32 rounding of the state only.
#include <atomic>
#include <cmath>

#include "fpb_common.cuh"

namespace fpb {
namespace {

struct CombineParams {
  float* seg;
  const void* start; int64_t start_sb, start_sh;
  int32_t n_seg, seg_len, T, H, reverse, state_f32;
  int64_t state_floats;
  float log2g[FPB_MAX_HEADS];
};

__device__ __forceinline__ float4 load4(const void* base, int64_t off, bool f32) {
  if (f32) return *reinterpret_cast<const float4*>((const float*)base + off);
  const uint2 raw = *reinterpret_cast<const uint2*>((const __nv_bfloat16*)base + off);
  const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
  const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
  return make_float4(a.x, a.y, b.x, b.y);
}
// grid (ceil(dk*dv / 4 / 256), H, B); one thread carries four adjacent state elements through the n pieces.  The local
// values do not depend on the running value: eight are loaded ahead of it (one ahead, the chain of round trips made the
// scan 5.2 us for 16 heads of 9 pieces).  Launched while the state-only pass still runs (programmatic dependent launch),
// as the walk is while the scan does: only the walk's start states wait for it.  The three launches of a prompt of 5003
// tokens, 16 heads, d = 128: 49.2 -> 45.1 us with the call around them.
__global__ void __launch_bounds__(256) segment_combine_kernel(const __grid_constant__ CombineParams p) {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int64_t e = ((int64_t)blockIdx.x * 256 + threadIdx.x) * 4;
  if (e >= p.state_floats) return;
  const int h = blockIdx.y, b = blockIdx.z;
  const float lg = p.log2g[h];
  float* seg = p.seg + ((int64_t)b * p.H + h) * p.n_seg * p.state_floats + e;
  float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
  if (p.start) a = load4(p.start, b * p.start_sb + h * p.start_sh + e, p.state_f32 != 0);
  auto piece = [&](int i) { return p.reverse ? p.n_seg - 1 - i : i; };
  auto slot_of = [&](int i) { return reinterpret_cast<float4*>(seg + (int64_t)piece(i) * p.state_floats); };
  constexpr int AHEAD = 8;
  for (int i0 = 0; i0 < p.n_seg; i0 += AHEAD) {
    float4 loc[AHEAD];
#pragma unroll
    for (int k = 0; k < AHEAD; ++k)                 // (the piece reached last has no local value: the walk itself ends it)
      if (i0 + k < p.n_seg - 1) loc[k] = *slot_of(i0 + k);
#pragma unroll
    for (int k = 0; k < AHEAD; ++k) {
      const int i = i0 + k;
      if (i < p.n_seg) *slot_of(i) = a;
      if (i < p.n_seg - 1) {
        const int len = min(p.seg_len, p.T - piece(i) * p.seg_len);
        const float g = exp2f((float)len * lg);
        a.x = fmaf(g, a.x, loc[k].x); a.y = fmaf(g, a.y, loc[k].y); a.z = fmaf(g, a.z, loc[k].z); a.w = fmaf(g, a.w, loc[k].w);
      }
    }
  }
}

}  // namespace

int sm_count() {
  static std::atomic<int> cache[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
  int n = cache[dev].load(std::memory_order_acquire);
  if (!n) {
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
    cache[dev].store(n, std::memory_order_release);
  }
  return n;
}

constexpr int kLongPiece = 512;          // tokens

// What a walk costs, in hundredths of a microsecond (fitted to one B200, 1 to 32 heads in all, d = 64 and 128, T = 300 to
// 32768): whole, 600 and 155 a chunk of its sequence; in pieces - state pass, scan and walk, three set-ups - 1400, 260 a chunk
// of a piece (`paired` where an SM gets two CTAs: kPairedChunk, less in the 64 x 128 tiles of the dQ walk) and 27 a piece, which
// the scan takes one after the other.  The two launches more are worth 600 of the host's time.  Both sides measured (forward,
// us): 8 heads, T = 1000, d = 128 whole 30.8, 8 pieces 22.7; 4 heads, T = 3000 in 5 pieces 41.1, in 24 26.3; but 16 heads,
// T = 600 whole 20.7, 4 pieces 24.7, 8 heads, T = 300 whole 13.7, 2 pieces 22.7, and 32 heads, T = 777, d = 64 whole 22.8, 7
// pieces 18.6, which a training call of 100 us of host work pays with 10 us.  (Pieces of at least 512 tokens, the rule before
// the launches were chained, left the first two at 30.8 and 41.1.)  Forward | backward by pieces: 1 head, d = 64, T = 8192 in 16
// 26.8 | 53.9, in 32 21.4 | 43.8, in 128 31.6 | 65.3, T = 32768 in 64 35.8 | 72.1, in 74 35.3 | 72.1, in 256 60.8 | 101; 2 heads,
// d = 128, T = 32768 in 64 48.3 | 106, in 74 55.0 | 119; 4 heads, d = 64, T = 8192 in 32 22.0 | 44.8, in 64 26.6 | 49.9; 16 heads
// in 8 44.5 | 89.3, in 16 38.2 | 83.3.
static long long cost_whole(int T) { return 600 + 155 * ((T + 63) / 64); }
static long long cost_pieces(int seg_len, long long count, long long a_chunk) { return 1400 + a_chunk * ((seg_len + 63) / 64) + 27 * count; }
constexpr int kLaunchesHost = 600;

Segments choose_segments(long long units, int ctas_per_sm, int T, int align, long long batch_heads, long long state_floats,
                         long long scratch_bytes, int B, int paired) {
  Segments none{1, 0};
  // Worth it only when the unsplit launch leaves at least half of the SMs without a CTA: with one CTA on (nearly) every
  // SM a second resident CTA adds little, and the first pass and the scan are not free (POP at B x H = 128, d = 64:
  // forward 0.189 ms whole, 0.204 ms in two pieces).
  const long long sms = sm_count();
  const long long slots = sms * ctas_per_sm;
  if (units <= 0 || units * 2 > sms || align <= 0) return none;
  long long most = slots / units;
  if (scratch_bytes > 0) {                                               // 0: the caller only asks how far a split would go
    const long long fit = scratch_bytes / (batch_heads * state_floats * 4);
    if (most > fit) most = fit;
  }
  if (B > 0 && most > 65535 / B) most = 65535 / B;                       // grid.z = batch x pieces
  auto cut = [&](long long shortest) {                                   // into as many pieces as allowed, each at least that long
    const long long n = most < T / shortest ? most : T / shortest;
    if (n < 2) return none;
    const int seg_len = (int)(((T + n - 1) / n + align - 1) / align) * align, count = (T + seg_len - 1) / seg_len;
    return count < 2 ? none : Segments{count, seg_len};
  };
  // the cheapest number of pieces (down to one `align` each; longer ones only cost more once their chunks outweigh all of it)
  Segments best = cut(align);
  if (best.n > 1) {
    constexpr int kAlone = 260;
    long long least = cost_pieces(best.seg_len, best.n, best.n * units > sms ? paired : kAlone);
    for (long long len = best.seg_len + align; len < T && cost_pieces((int)len, 0, kAlone) < least; len += align) {
      const long long count = (T + len - 1) / len, cost = cost_pieces((int)len, count, count * units > sms ? paired : kAlone);
      if (cost < least) { least = cost; best = Segments{(int)count, (int)len}; }
    }
    if (least + kLaunchesHost < cost_whole(T)) return best;
  }
  return cut(((kLongPiece + align - 1) / align) * align);                // pieces this long always paid
}

int launch_segment_combine(float* seg, Segments sg, int B, int T, int H, int dk, int dv, const float* gamma, bool reverse,
                           StateView start, bool state_f32, cudaStream_t stream) {
  CombineParams p;
  p.seg = seg;
  p.start = start.data; p.start_sb = start.sb; p.start_sh = start.sh;
  p.n_seg = sg.n; p.seg_len = sg.seg_len; p.T = T; p.H = H; p.reverse = reverse ? 1 : 0; p.state_f32 = state_f32 ? 1 : 0;
  p.state_floats = (int64_t)dk * dv;
  for (int h = 0; h < H; ++h) p.log2g[h] = (float)std::log2((double)gamma[h]);
  const dim3 grid((unsigned)((p.state_floats / 4 + 255) / 256), H, B);
  return launch_kernel(segment_combine_kernel, grid, 256, 0, true, p, stream) == cudaSuccess ? FPB_OK : FPB_ERR_LAUNCH;
}

}  // namespace fpb
