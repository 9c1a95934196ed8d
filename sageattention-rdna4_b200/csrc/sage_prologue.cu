// Quantisation prologue for B200: sequence mean of K (smooth_k; of V too with smooth_v), then one
// persistent, TMA-fed pass over the 128-token tiles of K, V and Q that writes the int8 / e4m3
// codes, the per-token scales and V transposed, and closes with the fold of the per-head S and its
// staged factor.  Short calls take one launch of clusters instead (quant_short_kernel).
//
// Arithmetic contract (reference: kernels/hip/h34_prologue.hip:116-211,259-282;
// kernels/hip/sk1_t6i.hip:104-117; kernels/hip/sk1_t4a1sb.hip:89-100;
// sageattention/sk1_backend/__init__.py:577-579).  Every operation below is a separate correctly
// rounded fp32 operation, written with the __f*_rn intrinsics so that no contraction or fast-math
// flag can change it:
//   mean  = f32( sum_n f64(K[n,d]) / f64(N) )
//   K     : x = f32(k) - mean; sk = max(amax/127, 1e-12); code = clamp(rne(x / sk), -128, 127)
//           e4m3 arm: sk = max(amax/448, 1e-12); code = e4m3(min(x / sk, 448))
//   V     : sv = max(amax/448, 1e-12); code = e4m3(min(v / sv, 448)); stored transposed
//   Q     : amax = max(amax, 1e-12); code = clamp(rint(q * (127/amax))); scale = amax/127
//           e4m3 arm: code = e4m3(clamp(q * (448/amax), +-448)); scale = amax/448
//   pad   : K8 = 0, SK = 1, V8T = 0, SV = 0
//   S     = max(max_n sv, 1); SVP = fl(fl(sv / S) * 448)
// The clamps to +-448 are done by the saturating e4m3 conversion (same codes).
// The fp64 mean is summed in a different (wider) order than the reference's eight strided
// partials; both are exact, hence identical, whenever the fp64 partial sums are exact, which holds
// for fp16 data when sum|K| < 2^29 per channel and for bf16 data of ordinary dynamic range.
#include <cuda.h>

#include <algorithm>
#include <type_traits>

#include "sage_common.cuh"
#include "sage_internal.h"

namespace sage {

constexpr int FOLD_KEYS = 4096;     // keys per fold item of the quantiser

// ------------------------------------------------------------------------------------------------
// Kernel 0: clears the control words (arrival counters, running maxima, status words, work and
// skip counters) of a call.  A kernel rather than a memset so that it and the mean kernel behind it
// can be launched as programmatic dependents: their CTAs are placed while the kernel before them
// on the stream drains, and the stream has no memset node to serialise on.
// ------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) clear_ctrl_kernel(unsigned* __restrict__ words, int n) {
  wait_for_predecessor();            // an earlier call may still be using these words
  allow_successor();
  for (int i = threadIdx.x; i < n; i += 256) words[i] = 0u;
}

// The same for a packed batch, and the batch's work list: the sequences ordered by their work,
// longest first, and in that order the prefix sums of their query tiles, key tiles, fold items and
// pairs of query tiles (plan: five arrays of B + 1 words).  The kernels behind it then draw only tiles that exist; in
// slots of the longest length, 59 % of the quantiser's items and of the attention grid were empty
// in a batch of eleven sequences of 512 .. 8 192 tokens.  One block: a few microseconds for up to
// PLAN_MAX_SEQS sequences.
__global__ void __launch_bounds__(PLAN_MAX_SEQS)
plan_packed_kernel(unsigned* __restrict__ words, int n, int* __restrict__ plan, int B,
                   const int* __restrict__ cu_q, const int* __restrict__ cu_k, long long Tq, long long Tk,
                   long long Nq, long long Nk) {
  __shared__ long long s_work[PLAN_MAX_SEQS];
  __shared__ int s_pre[4][PLAN_MAX_SEQS];
  wait_for_predecessor();
  allow_successor();
  const int tid = threadIdx.x;
  for (int i = tid; i < n; i += PLAN_MAX_SEQS) words[i] = 0u;
  // a sequence's live length, clamped to the packed tensor and to its slot as in the other kernels
  auto tiles = [&](const int* cu, long long T, long long cap) {
    const long long s0 = min(max((long long)cu[tid], 0LL), T), s1 = min((long long)cu[tid + 1], T);
    return (int)((min(max(s1 - s0, 0LL), cap) + TILE - 1) / TILE);
  };
  int tq = 0, tk = 0;
  if (tid < B) { tq = tiles(cu_q, Tq, Nq); tk = tiles(cu_k, Tk, Nk); }
  const long long work = (long long)tq * tk;
  s_work[tid] = work;
  s_pre[0][tid] = 0; s_pre[1][tid] = 0; s_pre[2][tid] = 0; s_pre[3][tid] = 0;
  __syncthreads();
  if (tid < B) {
    int rank = 0;
    for (int i = 0; i < B; ++i) rank += (s_work[i] > work || (s_work[i] == work && i < tid)) ? 1 : 0;
    plan[rank] = tid;
    s_pre[0][rank] = tq; s_pre[1][rank] = tk; s_pre[2][rank] = (tk * TILE + FOLD_KEYS - 1) / FOLD_KEYS;
    s_pre[3][rank] = (tq + 1) / 2;
  }
  __syncthreads();
  for (int off = 1; off < PLAN_MAX_SEQS; off <<= 1) {        // inclusive scan of the four arrays
    int v[4];
#pragma unroll
    for (int a = 0; a < 4; ++a) v[a] = (tid >= off) ? s_pre[a][tid - off] : 0;
    __syncthreads();
#pragma unroll
    for (int a = 0; a < 4; ++a) s_pre[a][tid] += v[a];
    __syncthreads();
  }
  if (tid < 4) plan[(tid + 1) * (B + 1)] = 0;
  if (tid < B)
#pragma unroll
    for (int a = 0; a < 4; ++a) plan[(a + 1) * (B + 1) + tid + 1] = s_pre[a][tid];
}

// ------------------------------------------------------------------------------------------------
// Kernel 1: partial fp64 column sums of K; the last CTA of a head combines them in split order.
// grid (nsplit, B*H), block 256 = 16 row lanes x 16 column chunks of 8 elements.
// ------------------------------------------------------------------------------------------------
template <typename T> struct MeanOf {   // one tensor: its rows, where its mean, partial sums and arrival counters are
  const T* x;
  float* mean;
  double* partial;
  unsigned* arrivals;
  long long sb, sh, sr;
};
// With smooth_v the means of K and V are one launch (blockIdx.z): each alone is mostly latency in
// calls of this size (4 x 16 heads, 2 048 x 64: two launches of 13 us).
template <typename T, bool VARLEN>
__global__ void __launch_bounds__(256)
kmean_kernel(const MeanOf<T> of_k, const MeanOf<T> of_v, long long N, long long H, int nsplit, long long chunk, int D,
             const int* __restrict__ cu, long long tokens) {
  const MeanOf<T>& of = (blockIdx.z == 0) ? of_k : of_v;
  const T* __restrict__ K = of.x;
  float* __restrict__ mean = of.mean;
  double* __restrict__ partial = of.partial;
  unsigned* __restrict__ arrivals = of.arrivals;
  const long long sb = of.sb, sh = of.sh, sr = of.sr;
  __shared__ double red[16][HD];
  __shared__ int s_last;
  wait_for_predecessor();            // the cleared arrival counters
  allow_successor();                 // (one wave, but for packed batches and for K and V together)
  const int tid = threadIdx.x, c = tid & 15, r = tid >> 4;
  const int split = blockIdx.x, bh = blockIdx.y;
  const long long b = bh / H, h = bh - b * H;
  const T* base = K + b * sb + h * sh + 8 * c;
  if (VARLEN) {                      // packed batch: this sequence's own length and first token
    // whatever the arrays hold, nothing outside the packed tokens is read
    const long long s0 = min(max((long long)cu[b], 0LL), tokens), s1 = min((long long)cu[b + 1], tokens);
    N = min(max(s1 - s0, 0LL), N);
    base = K + s0 * sr + h * sh + 8 * c;
  }
  const int n_arrive = VARLEN ? max((int)((N + chunk - 1) / chunk), 1) : nsplit;   // CTAs of this head with tokens
  if (VARLEN && split >= n_arrive) return;
  const long long n0 = (long long)split * chunk;
  const long long n1 = min(N, n0 + chunk);

  double acc[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) acc[e] = 0.0;
  const long long n_end = (8 * c < D) ? n1 : n0;   // columns past head_dim: nothing to read, mean 0
#pragma unroll 8
  for (long long n = n0 + r; n < n_end; n += 16) {
    const uint4 u = __ldcs(reinterpret_cast<const uint4*>(base + n * sr));   // streaming: read once here
    float x[8];
    unpack8<T>(u, x);
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[e] += (double)x[e];
  }
#pragma unroll
  for (int e = 0; e < 8; ++e) red[r][8 * c + e] = acc[e];
  __syncthreads();
  if (tid < HD) {
    double s = 0.0;
#pragma unroll
    for (int i = 0; i < 16; ++i) s += red[i][tid];
    partial[((size_t)bh * nsplit + split) * HD + tid] = s;
  }
  __threadfence();
  __syncthreads();
  if (tid == 0) s_last = (atomicAdd(&arrivals[bh], 1u) == (unsigned)(n_arrive - 1));
  __syncthreads();
  if (s_last && tid < HD) {
    __threadfence();
    double tot = 0.0;
    for (int sp = 0; sp < n_arrive; ++sp) tot += __ldcg(&partial[((size_t)bh * nsplit + sp) * HD + tid]);
    mean[(size_t)bh * HD + tid] = (!VARLEN || N > 0) ? (float)(tot / (double)N) : 0.f;
  }
}

// ------------------------------------------------------------------------------------------------
// Division.  K and V are divided by their scale with an IEEE-correct quotient obtained as
//   rc = rn(1/s) (correctly rounded);  q0 = rn(x*rc);  r = x - q0*s (one fma, exact);  q = fma(r, rc, q0)
// which equals rn(x/s) whenever rc is the correctly rounded reciprocal and nothing over/underflows
// (Markstein's theorem; |x/s| <= 448 and 1e-12 <= s here).  Three operations per element instead
// of a full division routine; checked against true division on 8e7 random samples on the host.
// Rounding to int8 uses the add-magic-constant trick (1.5*2^23): the addition rounds to nearest
// even, the low byte of the sum is the two's-complement code; |x/s| <= 127 needs no clamp.
// ------------------------------------------------------------------------------------------------
struct QuantArgs {
  uint8_t *q8, *k8, *v8t;
  float *sq, *sk, *sv, *svp, *s_fold;
  const float* mean;
  const float* vmean;             // optional: sequence mean of V, subtracted before quantising (smooth_v)
  unsigned* svmax_bits;           // per K/V head: running maximum of the V scales, as float bits
  unsigned* arrivals;             // per K/V head: V tiles whose scales are published
  long long N, N_pad, H;          // keys: length, padded length, K/V heads per batch element
  long long Nq, Hq, group;        // queries: length, heads per batch element, Hq / H (1 without GQA)
  long long BHq, BHkv;            // B*Hq, B*H
  float* qm;                      // optional (B*Hq, Nq): dot(q row, K mean of its K/V head), for the LSE
  int sub_mean;
  int32_t* status;                // set non-zero when a wait on a tile load ran out
  int32_t* status2;               // optional second word that receives the same report
  unsigned long long* next_item;  // global work counter (zeroed with the control block)
  const int *cu_q, *cu_k;         // VARLEN kernels: cumulative token counts of the packed batch (B + 1 entries each)
  long long Tq, Tk;               // VARLEN kernels: tokens in the packed q and k/v tensors
  const int* plan;                // VARLEN kernels, optional: the work list of plan_packed_kernel
  int n_seq;
  int only_q;                     // the K and V tiles are done (quant_short_kernel): Q tiles only
  long long drawn;                // items the work counter starts from: those that are done
};

// ------------------------------------------------------------------------------------------------
// Kernel 2: persistent CTAs (three per SM) draw 128-token tiles of K, V and Q from one global work
// counter; thread 0 keeps the next tile's 32 KB tensor-map load in flight into a shared-memory
// ring while the 256 threads quantise the tile that has landed.  Out-of-range rows and, for
// head_dim < 128, out-of-range columns arrive as zeros from the tensor map.
// Thread (c = tid & 7, r0 = tid >> 3) owns columns 8c..8c+7 and 64+8c..64+8c+7 of rows r0, r0+32,
// r0+64, r0+96: a quarter-warp reads one 256-byte row with two conflict-free 16-byte loads and the
// row maximum is three shuffles.
// Bound by HBM for long calls (48 heads x 47 520 tokens: 489 us, 2.6 GB), by instructions between the
// round trips otherwise: quotients for e4m3 two at a time, magnitudes on the packed 16-bit values,
// items worked out by one thread and one barrier less per item took 48 x 4 096 from 53 to 48 us, 24 x
// 27 280 (bf16) from 152 to 142 and 36 k packed tokens x 48 heads from 526 to 400.
// ------------------------------------------------------------------------------------------------
constexpr int QT_STAGES = 2;        // shared-memory ring: one tile being quantised, one in flight
constexpr int QT_MINBLOCKS = 3;     // CTAs per SM (3 x 64 KB of shared memory, 80 registers per thread)
constexpr uint32_t QT_STAGE_BYTES = TILE * HD * 2;
constexpr uint32_t QT_SMEM_BYTES = QT_STAGES * QT_STAGE_BYTES + 128 /* alignment slack */ + 64 /* barriers */;
constexpr long long QT_WAIT_CYCLES = 4000000000LL;

__device__ __forceinline__ uint32_t qt_smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t qt_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
               : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
  return ok;
}
__device__ __forceinline__ float quarter_warp_max(float x) {
  x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, 4));
  x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, 2));
  x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, 1));
  return x;
}
// rn(a / d) for a compile-time divisor: rc = rn(1/d) is a constant, the rest is Markstein's sequence
// (checked against true division over every mantissa of several binades for d = 127 and 448).
template <int DIV>
__device__ __forceinline__ float div_const(float a) {
  constexpr float d = (float)DIV, rc = 1.0f / (float)DIV;
  const float q0 = __fmul_rn(a, rc);
  const float r = __fmaf_rn(-q0, d, a);
  return __fmaf_rn(r, rc, q0);
}
__device__ __forceinline__ uint32_t i8x4_magic2(float2 ab, float2 cd) {
  const float2 m = make_float2(12582912.0f, 12582912.0f);
  const float2 u = __fadd2_rn(ab, m), v = __fadd2_rn(cd, m);
  return __byte_perm(__byte_perm(__float_as_uint(u.x), __float_as_uint(u.y), 0x0040),
                     __byte_perm(__float_as_uint(v.x), __float_as_uint(v.y), 0x0040), 0x5410);
}

// Largest magnitude of eight packed 16-bit values: exact on the packed form, half the instructions.
template <typename T> struct Packed16;
template <> struct Packed16<__half> { typedef __half2 Pair; };
template <> struct Packed16<__nv_bfloat16> { typedef __nv_bfloat162 Pair; };
template <typename T>
__device__ __forceinline__ float absmax16(const uint4& u, const uint4& v) {
  typedef typename Packed16<T>::Pair Pair;
  const uint32_t w[8] = {u.x, u.y, u.z, u.w, v.x, v.y, v.z, v.w};
  Pair m = __habs2(*reinterpret_cast<const Pair*>(&w[0]));
#pragma unroll
  for (int i = 1; i < 8; ++i) m = __hmax2(m, __habs2(*reinterpret_cast<const Pair*>(&w[i])));
  const float2 f = Elem<T>::cvt2(*reinterpret_cast<const uint32_t*>(&m));
  return fmaxf(f.x, f.y);
}
__device__ __forceinline__ float absmax3(float m, float2 x) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(m), "f"(fabsf(x.x)), "f"(fabsf(x.y)));
  return r;
}
// e4m3 codes of rn(x / s) for four values, given rc = rn(1/s).  The remainder is taken as q0*s - x and
// subtracted, which keeps the sign of a zero x; the packed operations have no negation, so the
// steps divide -x (all signs turn around, those of zeros too) and the codes' sign bits are flipped back.
__device__ __forceinline__ uint32_t e4m3x4_quot(float2 a, float2 b, float s, float rc) {
  const float2 nrc = make_float2(-rc, -rc), s2 = make_float2(s, s);
  const float2 qa = __fmul2_rn(a, nrc), qb = __fmul2_rn(b, nrc);
  const float2 ya = __ffma2_rn(__ffma2_rn(qa, s2, a), nrc, qa), yb = __ffma2_rn(__ffma2_rn(qb, s2, b), nrc, qb);
  return e4m3x4(ya.x, ya.y, yb.x, yb.y) ^ 0x80808080u;
}

// ------------------------------------------------------------------------------------------------
// One 128-token tile, already in shared memory (128 rows of 256 bytes), by 256 threads.  Thread
// (c = tid & 7, r0 = tid >> 3) owns columns 8c..8c+7 and 64+8c..64+8c+7 of rows r0, r0+32, r0+64,
// r0+96.  N: live tokens of the sequence.
// ------------------------------------------------------------------------------------------------
template <typename T, bool INT8>
__device__ __forceinline__ void quant_q_tile(const QuantArgs& a, const uint8_t* st, long long bh, long long n_base,
                                             long long N, int c, int r0) {
  constexpr float QMAX = INT8 ? I8_MAX : F8_MAX;
  constexpr int QDIV = INT8 ? 127 : 448;
  float mu[16];
  if (a.qm != nullptr) {
    const long long b = bh / a.Hq, h = bh - b * a.Hq, bh_kv = b * a.H + h / a.group;
#pragma unroll
    for (int e = 0; e < 8; ++e) { mu[e] = a.mean[(size_t)bh_kv * HD + 8 * c + e]; mu[8 + e] = a.mean[(size_t)bh_kv * HD + 64 + 8 * c + e]; }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int t = r0 + 32 * i;
    const long long nrow = n_base + t;
    float x[16];
    const uint4 u0 = *reinterpret_cast<const uint4*>(st + t * 256 + 16 * c), u1 = *reinterpret_cast<const uint4*>(st + t * 256 + 128 + 16 * c);
    unpack8<T>(u0, x);
    unpack8<T>(u1, x + 8);
    const float amax = fmaxf(quarter_warp_max(absmax16<T>(u0, u1)), SCALE_FLOOR);
    const float qinv = __fdiv_rn(QMAX, amax);
    float2 y[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) y[e] = make_float2(__fmul_rn(x[2 * e], qinv), __fmul_rn(x[2 * e + 1], qinv));
    uint2 w0, w1;
    if (INT8) {
      w0.x = i8x4_magic2(y[0], y[1]); w0.y = i8x4_magic2(y[2], y[3]);
      w1.x = i8x4_magic2(y[4], y[5]); w1.y = i8x4_magic2(y[6], y[7]);
    } else {
      w0.x = e4m3x4(y[0].x, y[0].y, y[1].x, y[1].y); w0.y = e4m3x4(y[2].x, y[2].y, y[3].x, y[3].y);
      w1.x = e4m3x4(y[4].x, y[4].y, y[5].x, y[5].y); w1.y = e4m3x4(y[6].x, y[6].y, y[7].x, y[7].y);
    }
    if (nrow < N) {
      uint8_t* dst = a.q8 + ((size_t)bh * a.Nq + nrow) * HD + 8 * c;
      *reinterpret_cast<uint2*>(dst) = w0;
      *reinterpret_cast<uint2*>(dst + 64) = w1;
      if (c == 0) a.sq[(size_t)bh * a.Nq + nrow] = div_const<QDIV>(amax);
    }
    if (a.qm != nullptr) {                          // fixed-order fp32 dot product of the raw row
      float d = 0.f;
#pragma unroll
      for (int e = 0; e < 16; ++e) d = __fmaf_rn(x[e], mu[e], d);
      d += __shfl_xor_sync(0xffffffffu, d, 4);
      d += __shfl_xor_sync(0xffffffffu, d, 2);
      d += __shfl_xor_sync(0xffffffffu, d, 1);
      if (c == 0 && nrow < N) a.qm[(size_t)bh * a.Nq + nrow] = d;
    }
  }
}

// mu: mean of K per column (read when a.sub_mean)
template <typename T, bool INT8>
__device__ __forceinline__ void quant_k_tile(const QuantArgs& a, const uint8_t* st, const float* mu, long long bh,
                                             long long n_base, long long N, int c, int r0) {
  constexpr int QDIV = INT8 ? 127 : 448;
  const long long N_pad = a.N_pad;
  float2 nmu[8];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const float* m0 = mu + 8 * c + 2 * e;
    nmu[e] = a.sub_mean ? make_float2(-m0[0], -m0[1]) : make_float2(0.f, 0.f);
    nmu[4 + e] = a.sub_mean ? make_float2(-m0[64], -m0[65]) : make_float2(0.f, 0.f);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int t = r0 + 32 * i;
    const long long nrow = n_base + t;
    const bool live = nrow < N;
    float x[16];
    unpack8<T>(*reinterpret_cast<const uint4*>(st + t * 256 + 16 * c), x);
    unpack8<T>(*reinterpret_cast<const uint4*>(st + t * 256 + 128 + 16 * c), x + 8);
    float2 xs[8];
    float amax = 0.f;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      xs[e] = __fadd2_rn(make_float2(x[2 * e], x[2 * e + 1]), nmu[e]);
      amax = absmax3(amax, xs[e]);
    }
    amax = quarter_warp_max(live ? amax : 0.f);
    const float sk = fmaxf(div_const<QDIV>(amax), SCALE_FLOOR);
    const float rc = __frcp_rn(sk);
    uint2 w0, w1;
    if (INT8) {
      // the sign of a zero quotient does not reach an int8 code, so the packed form is enough
      const float2 rc2 = make_float2(rc, rc), ns2 = make_float2(-sk, -sk);
      float2 y[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float2 q0 = __fmul2_rn(xs[e], rc2);
        const float2 r = __ffma2_rn(q0, ns2, xs[e]);
        y[e] = __ffma2_rn(r, rc2, q0);
      }
      w0.x = i8x4_magic2(y[0], y[1]); w0.y = i8x4_magic2(y[2], y[3]);
      w1.x = i8x4_magic2(y[4], y[5]); w1.y = i8x4_magic2(y[6], y[7]);
    } else {
      w0.x = e4m3x4_quot(xs[0], xs[1], sk, rc); w0.y = e4m3x4_quot(xs[2], xs[3], sk, rc);
      w1.x = e4m3x4_quot(xs[4], xs[5], sk, rc); w1.y = e4m3x4_quot(xs[6], xs[7], sk, rc);
    }
    if (!live) { w0 = make_uint2(0u, 0u); w1 = w0; }
    // rows are stored permuted inside 16-row blocks: key 4cc + jj of a block goes to row
    // 2cc + jj (jj < 2) or 8 + 2cc + jj - 2, the order in which the attention kernel's
    // 16-lane TMEM loads hand a thread four consecutive keys
    const long long o16 = nrow & 15, srow = (nrow & ~15LL) | ((o16 & 2) ? 8 + 2 * (o16 >> 2) + (o16 & 1) : 2 * (o16 >> 2) + (o16 & 1));
    uint8_t* dst = a.k8 + ((size_t)bh * N_pad + srow) * HD + 8 * c;
    *reinterpret_cast<uint2*>(dst) = w0;
    *reinterpret_cast<uint2*>(dst + 64) = w1;
    if (c == 0) a.sk[(size_t)bh * N_pad + nrow] = live ? sk : 1.0f;
  }
}

// The threads that share a tile: the whole block (BAR 0) or half of one (BAR 1 and 2).
template <int BAR> __device__ __forceinline__ void tile_sync() { asm volatile("bar.sync %0, 256;" ::"n"(BAR) : "memory"); }

// vmean: mean of V per column, or null.  The tile's scales also go to sv_tile, if given.  The stage is
// overwritten with the codes.  Returns this thread's largest scale of a live row.
template <typename T, bool VARLEN, int BAR>
__device__ __forceinline__ float quant_v_tile(const QuantArgs& a, uint8_t* st, const float* vmean, float* sv_tile, long long bh,
                                              long long n_base, long long N, int tid) {
  const int c = tid & 7, r0 = tid >> 3, lane = tid & 31, warp = tid >> 5;
  const long long N_pad = a.N_pad;
  float svmax = 0.f;
  uint2 w0[4], w1[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int t = r0 + 32 * i;
    const long long nrow = n_base + t;
    const bool live = nrow < N;
    float x[16];
    const uint4 u0 = *reinterpret_cast<const uint4*>(st + t * 256 + 16 * c), u1 = *reinterpret_cast<const uint4*>(st + t * 256 + 128 + 16 * c);
    unpack8<T>(u0, x);
    unpack8<T>(u1, x + 8);
    float amax;
    if (vmean) {
      amax = 0.f;
#pragma unroll
      for (int e = 0; e < 16; ++e) {
        x[e] = live ? __fsub_rn(x[e], vmean[(e < 8 ? 0 : 56) + 8 * c + e]) : 0.f;
        amax = fmaxf(amax, fabsf(x[e]));
      }
    } else {
      amax = absmax16<T>(u0, u1);
      if (VARLEN && !live) {                               // the rows behind a packed sequence are its neighbour's
        amax = 0.f;
#pragma unroll
        for (int e = 0; e < 16; ++e) x[e] = 0.f;
      }
    }
    amax = quarter_warp_max(amax);
    const float sv = fmaxf(div_const<448>(amax), SCALE_FLOOR);
    const float rc = __frcp_rn(sv);
    const float2* x2 = reinterpret_cast<const float2*>(x);
    w0[i].x = e4m3x4_quot(x2[0], x2[1], sv, rc); w0[i].y = e4m3x4_quot(x2[2], x2[3], sv, rc);
    w1[i].x = e4m3x4_quot(x2[4], x2[5], sv, rc); w1[i].y = e4m3x4_quot(x2[6], x2[7], sv, rc);
    if (c == 0) {
      a.sv[(size_t)bh * N_pad + nrow] = live ? sv : 0.0f;
      if (sv_tile) sv_tile[t] = live ? sv : 0.0f;
      if (live) svmax = fmaxf(svmax, sv);
    }
  }
  tile_sync<BAR>();                // every thread has read its rows: the stage becomes the code tile
  uint32_t* vt = reinterpret_cast<uint32_t*>(st);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int t = r0 + 32 * i;
    const int key = (((t >> 4) & 7) << 2) ^ ((t & 1) << 4);
    *reinterpret_cast<uint2*>(&vt[t * 32 + ((2 * c) ^ key)]) = w0[i];
    *reinterpret_cast<uint2*>(&vt[t * 32 + ((16 + 2 * c) ^ key)]) = w1[i];
  }
  tile_sync<BAR>();
  {
    const int tg = lane & 7, dq = 4 * warp + (lane >> 3);
    uint32_t o[4][4];
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      const int tk = 16 * tg + 4 * g;
      const uint32_t w0_ = vt[(tk + 0) * 32 + (dq ^ (tg << 2))];
      const uint32_t w1_ = vt[(tk + 1) * 32 + (dq ^ (tg << 2) ^ 16)];
      const uint32_t w2_ = vt[(tk + 2) * 32 + (dq ^ (tg << 2))];
      const uint32_t w3_ = vt[(tk + 3) * 32 + (dq ^ (tg << 2) ^ 16)];
      const uint32_t t0 = __byte_perm(w0_, w1_, 0x5140), t1 = __byte_perm(w2_, w3_, 0x5140);
      const uint32_t t2 = __byte_perm(w0_, w1_, 0x7362), t3 = __byte_perm(w2_, w3_, 0x7362);
      o[0][g] = __byte_perm(t0, t1, 0x5410);
      o[1][g] = __byte_perm(t0, t1, 0x7632);
      o[2][g] = __byte_perm(t2, t3, 0x5410);
      o[3][g] = __byte_perm(t2, t3, 0x7632);
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      uint8_t* dst = a.v8t + ((size_t)bh * HD + 4 * dq + e) * N_pad + n_base + 16 * tg;
      *reinterpret_cast<uint4*>(dst) = make_uint4(o[e][0], o[e][1], o[e][2], o[e][3]);
    }
  }
  return svmax;
}

// VARLEN: a packed batch.  N, N_pad and Nq are then the capacity of a sequence's slot in the outputs
// (sized for the longest sequence allowed); every sequence has its own length and its own first
// token in the inputs, read from cu_q / cu_k.  Tiles past a sequence's end are neither loaded nor
// written (the attention kernel never visits them).
template <typename T, bool INT8, bool VARLEN>
__global__ void __launch_bounds__(256, QT_MINBLOCKS)
quant_qkv_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                     const __grid_constant__ CUtensorMap tm_v, const QuantArgs a) {
  extern __shared__ uint8_t qt_smem[];
  __shared__ int4 s_item[QT_STAGES];   // what the stage holds: {tensor (0 q, 1 k, 2 v, 3 a fold, -1 the end), head, tile, live tokens}
  __shared__ int s_drawn;              // thread 0's next item (in a register it makes the int8 kernels spill)
  __shared__ int s_plan[VARLEN ? 4 * (PLAN_MAX_SEQS + 1) : 1];
  const uint32_t raw_addr = qt_smem_u32(qt_smem);
  const uint32_t base = (raw_addr + 127u) & ~127u;
  uint8_t* gbase = qt_smem + (base - raw_addr);
  const uint32_t bar0 = base + QT_STAGES * QT_STAGE_BYTES;
  const int tid = threadIdx.x, c = tid & 7, r0 = tid >> 3, lane = tid & 31, warp = tid >> 5;

  if (tid == 0) {
    for (int s = 0; s < QT_STAGES; ++s)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar0 + 8u * (uint32_t)s), "r"(1u) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  wait_for_predecessor();            // the means and the cleared control block
  allow_successor();                 // persistent grid: every CTA is resident

  const bool planned = VARLEN && a.plan != nullptr;
  const int P1 = VARLEN ? a.n_seq + 1 : 0;
  if (planned) {
    for (int i = tid; i < 4 * P1; i += 256) s_plan[i] = a.plan[i];
    __syncthreads();
  }
  // Counts of items fit 32 bits: every K, V or Q item stands for 16 KB of codes.
  const int tiles_q = (int)((a.Nq + TILE - 1) / TILE), tiles_k = (int)(a.N_pad / TILE);
  const int fold_per_head = (int)((a.N_pad + FOLD_KEYS - 1) / FOLD_KEYS);
  const int items_k = a.only_q ? 0 : planned ? s_plan[3 * P1 - 1] * (int)a.H : (int)a.BHkv * tiles_k;
  const int items_q = planned ? s_plan[2 * P1 - 1] * (int)a.Hq : (int)a.BHq * tiles_q;
  const int items_f = a.only_q ? 0 : planned ? s_plan[4 * P1 - 1] * (int)a.H : (int)a.BHkv * fold_per_head;
  const int total = 2 * items_k + items_q + items_f;

  // item -> (tensor, head, tile): K first with the last heads first (their rows are still in L2
  // after the mean pass), then V (so that the per-head folds overlap the Q items), then Q, then the
  // folds.  With a work list: sequence by sequence in the list's order, head by head.
  auto decode = [&](int it, int& which, int& bh, int& tile) {
    int j = it;
    if (it < items_k) which = 1;
    else if (it < 2 * items_k) { which = 2; j -= items_k; }
    else if (it < 2 * items_k + items_q) { which = 0; j -= 2 * items_k; }
    else { which = 3; j -= 2 * items_k + items_q; }
    if (planned) {
      const int heads = (int)((which == 0) ? a.Hq : a.H);
      const int* pre = s_plan + (which == 0 ? 1 : which == 3 ? 3 : 2) * P1;
      int lo = 0, hi = a.n_seq;        // pre[lo] * heads <= j < pre[hi] * heads
      while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (pre[mid] * heads <= j) lo = mid; else hi = mid;
      }
      const int rem = j - pre[lo] * heads, per = pre[lo + 1] - pre[lo];
      bh = s_plan[lo] * heads + rem / per;
      tile = rem % per;
    } else {
      const int per = (which == 0) ? tiles_q : which == 3 ? fold_per_head : tiles_k;
      const int r = j / per;
      bh = (int)((which == 0) ? a.BHq : a.BHkv) - 1 - r;
      tile = j - r * per;
    }
  };
  // length and first input token of the sequence an item belongs to
  auto seq_of = [&](int which, int bh, long long& start) -> long long {
    if (!VARLEN) { start = 0; return (which == 0) ? a.Nq : a.N; }
    const int b = bh / (int)((which == 0) ? a.Hq : a.H);
    const int* cu = (which == 0) ? a.cu_q : a.cu_k;
    // clamped to the packed tensor: whatever the arrays hold, a sequence lies inside it
    const long long T = (which == 0) ? a.Tq : a.Tk;
    const long long s0 = min(max((long long)__ldg(cu + b), 0LL), T), s1 = min((long long)__ldg(cu + b + 1), T);
    start = s0;
    return min(max(s1 - s0, 0LL), (which == 0) ? a.Nq : a.N);
  };
  // Items are handed out through one global counter: a CTA that is held up (by a head's fold, say)
  // simply takes fewer of them.  Thread 0 draws an item, works out what it is, publishes that in
  // s_item and starts the load; the other threads see it with the stage's barrier.  The counter is
  // drawn one item ahead, so the atomic's round trip is off the critical path.
  auto draw = [&]() { return (int)((long long)atomicAdd(a.next_item, 1ULL) - a.drawn); };
  auto issue = [&](int stage, int it) {
    const uint32_t bar_ = bar0 + 8u * (uint32_t)stage;
    int which = -1, bh = 0, tile = 0;
    long long start = 0, len = 0;
    if (it < total) {
      decode(it, which, bh, tile);
      len = seq_of(which == 3 ? 1 : which, bh, start);
    }
    s_item[stage] = make_int4(which, bh, tile, (int)len);
    // the end, folds and tiles past their sequence's end load nothing
    if (which < 0 || which == 3 || (VARLEN && (long long)tile * TILE >= len)) {
      asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar_) : "memory");
      return;
    }
    const int heads = (int)((which == 0) ? a.Hq : a.H);
    const int b = VARLEN ? 0 : bh / heads, h = bh % heads;        // (a packed batch's map has one batch entry)
    const long long row = start + (long long)tile * TILE;
    const CUtensorMap* map = (which == 0) ? &tm_q : (which == 1 ? &tm_k : &tm_v);
    const uint32_t bar = bar0 + 8u * (uint32_t)stage, dst = base + (uint32_t)stage * QT_STAGE_BYTES;
    // the stage was last touched by ordinary loads and stores (V tiles are staged back into it);
    // order them before the copy engine's writes
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(QT_STAGE_BYTES) : "memory");
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
        ::"r"(dst), "l"(map), "r"(bar), "r"(0), "r"((int)row), "r"(h), "r"(b) : "memory");
  };

  __syncthreads();
  if (tid == 0) {
    for (int p = 0; p < QT_STAGES - 1; ++p) issue(p, draw());
    s_drawn = draw();
  }
  __syncthreads();                     // s_item of the first stage, for a thread whose wait runs out too

  for (uint32_t n = 0;; ++n) {
    const int stage = (int)(n % QT_STAGES);
    const uint32_t parity = (n / QT_STAGES) & 1u;
    if (tid == 0) {                    // into the stage released by the previous item
      issue((int)((n + QT_STAGES - 1) % QT_STAGES), s_drawn);
      s_drawn = draw();                // consumed one iteration later
    }
    // bounded wait for this item's tile; a thread that gives up goes on to the barrier at the end of
    // the item, where all leave together
    int lost = 0;
    {
      const uint32_t bar = bar0 + 8u * (uint32_t)stage;
      if (!qt_try_wait(bar, parity)) {
        const long long t0 = clock64();
        uint32_t spins = 0;
        while (!qt_try_wait(bar, parity)) {
          if ((++spins & 1023u) == 0u && clock64() - t0 > QT_WAIT_CYCLES) { lost = 1; break; }
        }
      }
    }
    const int4 item = s_item[stage];
    const int which = item.x;
    if (which < 0) break;              // the list is exhausted (every thread reads the same value)
    const int bh = item.y, tile = item.z, seq_len = item.w;
    const long long n_base = (long long)tile * TILE;
    const uint8_t* st = gbase + (size_t)stage * QT_STAGE_BYTES;
    const bool beyond = VARLEN && which != 3 && n_base >= seq_len;   // nothing was loaded, nothing is written

    if (beyond) {
    } else if (which == 0) {
      // ---------------------------------- Q ----------------------------------
      const long long N = VARLEN ? seq_len : a.Nq;
      quant_q_tile<T, INT8>(a, st, bh, n_base, N, c, r0);
    } else if (which == 1) {
      // ---------------------------------- K ----------------------------------
      const long long N = VARLEN ? seq_len : a.N;
      quant_k_tile<T, INT8>(a, st, a.mean + (size_t)bh * HD, bh, n_base, N, c, r0);
    } else if (which == 2) {
      // ---------------------------------- V ----------------------------------
      const long long N = VARLEN ? seq_len : a.N;
      float svmax = quant_v_tile<T, VARLEN, 0>(a, gbase + (size_t)stage * QT_STAGE_BYTES, a.vmean ? a.vmean + (size_t)bh * HD : nullptr,
                                               nullptr, bh, n_base, N, tid);
      // per-head max of the V scale (all scales are >= 0, so the unsigned order of the bit patterns
      // is the float order); S and SVP are folded by the closing items of the list
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) svmax = fmaxf(svmax, __shfl_xor_sync(0xffffffffu, svmax, off));
      if (lane == 0 && svmax > 0.f) atomicMax(&a.svmax_bits[bh], __float_as_uint(svmax));
    } else if (which == 3) {
      // ------------------------- fold of one head's V scales -------------------------
      // S = max(max sv, 1), SVP = fl(fl(sv / S) * 448) for FOLD_KEYS keys (the reference's
      // fold_v_scale and the attention kernel's staging).  These items close the list, long after
      // the head's V tiles were drawn; thread 0 still waits, bounded, for their arrivals.
      int done = 1;
      if (tid == 0) {
        const unsigned want = VARLEN ? (unsigned)((seq_len + TILE - 1) / TILE) : (unsigned)tiles_k;
        const volatile unsigned* arr = a.arrivals + bh;
        if (*arr != want) {
          const long long t0 = clock64();
          while (*arr != want) {
            if (clock64() - t0 > QT_WAIT_CYCLES) { done = 0; break; }
          }
        }
        __threadfence();               // acquire: the V scales of every arrived tile are visible
      }
      if (!__syncthreads_and(done)) {
        if (tid == 0) { atomicOr(a.status, 2); if (a.status2) atomicOr(a.status2, 8); }
        break;
      }
      const long long N_pad = a.N_pad;
      const long long n_fold = VARLEN ? ((long long)seq_len + TILE - 1) / TILE * TILE : N_pad;   // rows that were written
      const float S = fmaxf(__uint_as_float(__ldcg(&a.svmax_bits[bh])), 1.0f);
      if (tile == 0 && tid == 0) a.s_fold[bh] = S;
#pragma unroll
      for (int i = 0; i < FOLD_KEYS / 1024; ++i) {
        const long long nn = (long long)tile * FOLD_KEYS + i * 1024 + 4 * tid;
        if (nn < n_fold) {             // a multiple of 128: whole float4s
          const float4 v = __ldcg(reinterpret_cast<const float4*>(a.sv + (size_t)bh * N_pad + nn));
          float4 o;
          o.x = __fmul_rn(__fdiv_rn(v.x, S), F8_MAX); o.y = __fmul_rn(__fdiv_rn(v.y, S), F8_MAX);
          o.z = __fmul_rn(__fdiv_rn(v.z, S), F8_MAX); o.w = __fmul_rn(__fdiv_rn(v.w, S), F8_MAX);
          *reinterpret_cast<float4*>(a.svp + (size_t)bh * N_pad + nn) = o;
        }
      }
    }
    if (__syncthreads_or(lost)) {      // the stage may be refilled
      if (tid == 0) { atomicOr(a.status, 1); if (a.status2) atomicOr(a.status2, 8); }
      const long long t0 = clock64();
      while (clock64() - t0 < 400000) { }     // give copies still in flight a moment to land
      break;
    }
    if (which == 2 && !beyond && tid == 0) {   // this tile's V scales and maximum are published: one release per CTA
      __threadfence();
      atomicAdd(a.arrivals + bh, 1u);
    }
  }
}

// ------------------------------------------------------------------------------------------------
// Short key sequences (at most SHORT_CTAS tiles): the whole prologue in one launch.  The CTAs of a
// cluster hold the K and V tiles of one K/V head in their shared memory, one of each per CTA.  Half of a CTA's threads sum the K tiles' columns, hand the sums to the other CTAs through
// distributed shared memory, and quantise with the mean of all; the other half quantises V, and the
// largest V scale of the cluster gives S.  K is read once, there are no control words to clear, no
// work counter and no fold items: such calls spend their time on launches and round trips to
// memory, not on bandwidth.  48 heads of 288 tokens: three launches of 17 us in all before, one of
// 10 us now.
// Further clusters take the Q tiles, one per half.
// ------------------------------------------------------------------------------------------------
struct ShortArgs {
  float *mean, *vmean;
  unsigned* words;                // control words, cleared here for the kernels behind this one
  int n_words, kv_clusters;
  int counter_word;               // the work counter, which is set to the number of tiles done here
  unsigned items;
  long long items_q;
};
constexpr int SHORT_CTAS = 16;    // the largest cluster, with two CTAs on an SM
namespace short_smem {
constexpr uint32_t RED = 2 * QT_STAGE_BYTES;                    // [2][4][128] fp64: column sums of warps
constexpr uint32_t PART = RED + 2 * 4 * HD * 8;                 // [2][SHORT_CTAS][128] fp64: column sums of CTAs
constexpr uint32_t MEAN = PART + 2 * SHORT_CTAS * HD * 8;       // [2][128] fp32
constexpr uint32_t SV = MEAN + 2 * HD * 4;                      // [128] fp32: V scales
constexpr uint32_t BARS = SV + TILE * 4;
constexpr uint32_t SVMAX = BARS + 2 * 8;
constexpr uint32_t BYTES = SVMAX + 16 + 128 /* alignment slack */;
static_assert(2 * (BYTES + 1024) <= 228 * 1024, "two CTAs share an SM");
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
__device__ __forceinline__ uint32_t in_cta(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}

template <typename T, bool INT8>
__global__ void __launch_bounds__(512, 2)
quant_short_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                   const __grid_constant__ CUtensorMap tm_v, const QuantArgs a, const ShortArgs sa) {
  namespace L = short_smem;
  extern __shared__ uint8_t qt_smem[];
  const uint32_t raw_addr = qt_smem_u32(qt_smem), base = (raw_addr + 127u) & ~127u;
  uint8_t* gbase = qt_smem + (base - raw_addr);
  const int tid = threadIdx.x, grp = tid >> 8, gt = tid & 255, lane = tid & 31, gwarp = gt >> 5;
  const int c = gt & 7, r0 = gt >> 3;
  uint32_t C, rank;
  asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(C));
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  const int cluster = (int)(blockIdx.x / C);
  const uint32_t bar = base + L::BARS + 8u * (uint32_t)grp;          // this half's tile
  volatile unsigned* svmax_s = reinterpret_cast<volatile unsigned*>(gbase + L::SVMAX);
  if (tid == 0) {
    for (int i = 0; i < 2; ++i)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(base + L::BARS + 8u * (uint32_t)i), "r"(1u) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    *svmax_s = 0u;
  }
  __syncthreads();
  cluster_arrive();
  cluster_wait();                    // every CTA of the cluster runs: its shared memory may be written
  wait_for_predecessor();            // an earlier call may still be using the buffers
  allow_successor();
  if (blockIdx.x == 0)
    for (int i = tid; i < sa.n_words; i += 512) sa.words[i] = (i == sa.counter_word) ? sa.items : 0u;

  auto load = [&](const CUtensorMap* map, long long tile, long long bh, long long heads) {
    const uint32_t dst = base + (uint32_t)grp * QT_STAGE_BYTES;
    const int b = (int)(bh / heads), h = (int)(bh - (long long)b * heads);
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(QT_STAGE_BYTES) : "memory");
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
        ::"r"(dst), "l"(map), "r"(bar), "r"(0), "r"((int)(tile * TILE)), "r"(h), "r"(b) : "memory");
  };
  // bounded wait; a thread that gives up reports it and goes on, so that no barrier misses it.  It does
  // not wait a second time, and it stays a moment before it leaves: the copy may still arrive, and this
  // CTA's shared memory must not be another's by then.
  bool lost = false;
  auto landed = [&]() {
    if (lost || qt_try_wait(bar, 0)) return;
    const long long t0 = clock64();
    while (!qt_try_wait(bar, 0))
      if (clock64() - t0 > QT_WAIT_CYCLES) { atomicOr(a.status, 1); if (a.status2) atomicOr(a.status2, 8); lost = true; return; }
  };
  auto before_leaving = [&]() {
    if (lost) {
      const long long t0 = clock64();
      while (clock64() - t0 < 400000) { }
    }
  };
  uint8_t* stage = gbase + (uint32_t)grp * QT_STAGE_BYTES;
  auto half_sync = [&]() { if (grp == 0) tile_sync<1>(); else tile_sync<2>(); };

  if (cluster >= sa.kv_clusters) {   // Q tiles
    const long long tiles_q = (a.Nq + TILE - 1) / TILE;
    const long long item = ((long long)(cluster - sa.kv_clusters) * C + rank) * 2 + grp;
    if (item >= sa.items_q) return;
    const long long bh = item / tiles_q, tile = item - bh * tiles_q;
    if (gt == 0) load(&tm_q, tile, bh, a.Hq);
    landed();
    quant_q_tile<T, INT8>(a, stage, bh, tile * TILE, a.Nq, c, r0);
    before_leaving();
    return;
  }

  const long long bh = cluster, n_base = (long long)rank * TILE;      // tile `rank` of both tensors
  if (gt == 0) load(grp == 0 ? &tm_k : &tm_v, rank, bh, a.H);
  const bool has_mean = (grp == 0) ? a.sub_mean != 0 : sa.vmean != nullptr;
  float* mean_s = reinterpret_cast<float*>(gbase + L::MEAN) + grp * HD;
  if (has_mean) {
    // column sums in fp64 (exact for fp16 values, see the top of the file): rows by half-warps,
    // then warps, then CTAs, all in a fixed order
    const int cc = gt & 15, rr = gt >> 4;
    double acc[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[e] = 0.0;
    landed();
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      float x[8];
      unpack8<T>(*reinterpret_cast<const uint4*>(stage + (rr + 16 * k) * 256 + 16 * cc), x);
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[e] += (double)x[e];
    }
    double* red = reinterpret_cast<double*>(gbase + L::RED) + grp * 4 * HD + (gwarp & 3) * HD + 8 * cc;
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[e] += __shfl_xor_sync(0xffffffffu, acc[e], 16);
    if (gwarp >= 4 && lane < 16)
#pragma unroll
      for (int e = 0; e < 8; ++e) red[e] = acc[e];
    half_sync();
    if (gwarp < 4 && lane < 16)
#pragma unroll
      for (int e = 0; e < 8; ++e) red[e] += acc[e];
    half_sync();
    if (gt < HD) {
      const double* col = reinterpret_cast<const double*>(gbase + L::RED) + grp * 4 * HD + gt;
      const double t = (col[0] + col[HD]) + (col[2 * HD] + col[3 * HD]);
      const uint32_t at = base + L::PART + (uint32_t)((grp * SHORT_CTAS + rank) * HD + gt) * 8u;
      for (uint32_t r = 0; r < C; ++r)
        asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(in_cta(at, r)), "d"(t) : "memory");
    }
  }
  float svmax = 0.f;
  float* sv_s = reinterpret_cast<float*>(gbase + L::SV);
  auto quant_v = [&](const float* vmean) {
    landed();
    svmax = quant_v_tile<T, false, 2>(a, stage, vmean, sv_s, bh, n_base, a.N, gt);
  };
  cluster_arrive();                  // this CTA's column sums are with the others
  if (grp == 1 && !has_mean) quant_v(nullptr);
  cluster_wait();
  if (has_mean) {
    if (gt < HD) {
      const double* part = reinterpret_cast<const double*>(gbase + L::PART) + grp * SHORT_CTAS * HD;
      double t = 0.0;
      for (uint32_t r = 0; r < C; ++r) t += part[r * HD + gt];
      const float m = (float)(t / (double)a.N);
      mean_s[gt] = m;
      if (rank == 0) (grp == 0 ? sa.mean : sa.vmean)[(size_t)bh * HD + gt] = m;
    }
    half_sync();
  }
  if (grp == 0) {
    landed();
    quant_k_tile<T, INT8>(a, stage, mean_s, bh, n_base, a.N, c, r0);
  } else {
    if (has_mean) quant_v(mean_s);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) svmax = fmaxf(svmax, __shfl_xor_sync(0xffffffffu, svmax, off));
    if (lane < (int)C)               // non-negative floats order like their bits
      asm volatile("red.relaxed.cluster.shared::cluster.max.u32 [%0], %1;"
                   ::"r"(in_cta(base + L::SVMAX, (uint32_t)lane)), "r"(__float_as_uint(svmax)) : "memory");
  }
  cluster_arrive();
  cluster_wait();                    // the head's largest V scale is complete
  if (grp == 1) {
    const float S = fmaxf(__uint_as_float(*svmax_s), 1.0f);
    if (rank == 0 && gt == 0) a.s_fold[bh] = S;
    if (gt < TILE) a.svp[(size_t)bh * a.N_pad + n_base + gt] = __fmul_rn(__fdiv_rn(sv_s[gt], S), F8_MAX);
  }
  before_leaving();
}

// ------------------------------------------------------------------------------------------------
// Host launcher.
// ------------------------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                                  CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                  CUtensorMapFloatOOBfill);
static EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  }
  return fn;
}
// 4-D map over a logical (B, H, N, D) view of 2-byte elements with (batch, head, row) element
// strides: box 128 columns x 128 rows, no swizzle, out-of-range elements read as zero.
static bool make_map4(CUtensorMap* m, const void* ptr, CUtensorMapDataType dt, int64_t D, int64_t N, int64_t H,
                      int64_t B, const int64_t strides_bhr[3]) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return false;
  cuuint64_t dims[4] = {(cuuint64_t)D, (cuuint64_t)N, (cuuint64_t)H, (cuuint64_t)B};
  cuuint64_t strides[3] = {(cuuint64_t)strides_bhr[2] * 2, (cuuint64_t)strides_bhr[1] * 2, (cuuint64_t)strides_bhr[0] * 2};
  cuuint32_t box[4] = {128, 128, 1, 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  return fn(m, dt, 4, const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

static cudaLaunchConfig_t short_config(cudaLaunchAttribute attr[2], unsigned clusters, unsigned ctas, cudaStream_t st) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(clusters * ctas); cfg.blockDim = dim3(512); cfg.dynamicSmemBytes = short_smem::BYTES; cfg.stream = st;
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = ctas; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr; cfg.numAttrs = 2;
  return cfg;
}

// The largest cluster of quant_short_kernel that the device can place (16, 8 or none; a partition of
// a GPU may have fewer SMs side by side), asked once per device together with the opt-ins.
template <typename T, bool INT8>
static cudaError_t short_cluster_limit(int dev, int* limit) {
  static int known[64] = {0};                                           // limit + 1
  if (known[dev] == 0) {
    auto kern = quant_short_kernel<T, INT8>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)short_smem::BYTES);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return e;
    int best = 0;
    for (int ctas = SHORT_CTAS; ctas >= 8 && best == 0; ctas /= 2) {
      cudaLaunchAttribute attr[2];
      cudaLaunchConfig_t cfg = short_config(attr, 1, (unsigned)ctas, nullptr);
      cfg.attrs = attr + 1; cfg.numAttrs = 1;                           // the cluster size alone
      int n = 0;
      if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) == cudaSuccess && n > 0) best = ctas;
      else (void)cudaGetLastError();
    }
    known[dev] = best + 1;
  }
  *limit = known[dev] - 1;
  return cudaSuccess;
}

template <typename T, bool INT8>
static cudaError_t launch_short(const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv, const QuantArgs& a,
                                const ShortArgs& sa, int64_t tiles_k, cudaStream_t st) {
  const unsigned ctas = (unsigned)tiles_k;                              // per cluster
  const int64_t per_cluster = (int64_t)ctas * 2;                        // Q tiles a cluster takes
  const unsigned clusters = (unsigned)(sa.kv_clusters + (sa.items_q + per_cluster - 1) / per_cluster);
  cudaLaunchAttribute attr[2];
  const cudaLaunchConfig_t cfg = short_config(attr, clusters, ctas, st);
  return cudaLaunchKernelEx(&cfg, quant_short_kernel<T, INT8>, mq, mk, mv, a, sa);
}

template <typename T>
static cudaError_t launch_typed(const PrologueParams& p, cudaStream_t st) {
  const int64_t bh = p.B * p.H;
  unsigned* words = reinterpret_cast<unsigned*>(p.ctrl);
  double* partial = reinterpret_cast<double*>(reinterpret_cast<char*>(p.ctrl) + CtrlHeader::partial_off(bh));
  // SM count and the opt-in to 64 KB of dynamic shared memory: looked up once per device
  static int sm_count[64] = {0};
  static bool opted_in[64][4] = {{false}};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  if (sm_count[dev] == 0) {
    e = cudaDeviceGetAttribute(&sm_count[dev], cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
  }
  QuantArgs a;
  a.q8 = reinterpret_cast<uint8_t*>(p.q8); a.k8 = reinterpret_cast<uint8_t*>(p.k8);
  a.v8t = reinterpret_cast<uint8_t*>(p.v8t);
  a.sq = p.sq; a.sk = p.sk; a.sv = p.sv; a.svp = p.svp; a.s_fold = p.s_fold; a.mean = p.mean; a.vmean = p.vmean;
  a.svmax_bits = words + 2 * bh; a.arrivals = words + bh;
  a.N = p.N; a.N_pad = p.N_pad; a.H = p.H;
  a.Nq = p.Nq; a.Hq = p.Hq; a.group = p.Hq / p.H; a.BHq = p.B * p.Hq; a.BHkv = bh; a.qm = p.qm;
  a.sub_mean = p.smooth_k ? 1 : 0;
  a.cu_q = p.cu_q; a.cu_k = p.cu_k; a.Tq = p.Tq; a.Tk = p.Tk;
  a.plan = p.plan; a.n_seq = (int)p.B; a.only_q = 0; a.drawn = 0;
  const bool varlen = p.cu_q != nullptr;
  const int64_t tq = (p.Nq + TILE - 1) / TILE, tk = p.N_pad / TILE;
  a.status = reinterpret_cast<int32_t*>(words + CtrlHeader::status_word(bh));
  a.status2 = p.status;
  a.next_item = reinterpret_cast<unsigned long long*>(words + CtrlHeader::status_word(bh) + 2);
  CUtensorMap mq, mk, mv;
  const CUtensorMapDataType dt = (sizeof(T) == 2 && std::is_same<T, __half>::value) ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16
                                                                                      : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  if (varlen) {
    // packed (tokens, heads, D) tensors: one batch entry that holds every token
    const int64_t qs[3] = {p.q_strides[1], p.q_strides[1], p.q_strides[2]};
    const int64_t ks[3] = {p.k_strides[1], p.k_strides[1], p.k_strides[2]};
    const int64_t vs[3] = {p.v_strides[1], p.v_strides[1], p.v_strides[2]};
    if (!make_map4(&mq, p.q, dt, p.D, p.Tq, p.Hq, 1, qs) || !make_map4(&mk, p.k, dt, p.D, p.Tk, p.H, 1, ks) ||
        !make_map4(&mv, p.v, dt, p.D, p.Tk, p.H, 1, vs))
      return cudaErrorInvalidValue;
  } else if (!make_map4(&mq, p.q, dt, p.D, p.Nq, p.Hq, p.B, p.q_strides) ||
             !make_map4(&mk, p.k, dt, p.D, p.N, p.H, p.B, p.k_strides) ||
             !make_map4(&mv, p.v, dt, p.D, p.N, p.H, p.B, p.v_strides))
    return cudaErrorInvalidValue;
  // Short calls take one launch, see quant_short_kernel.  Its CTAs do one tile each and wait for
  // each other, so that it pays while there are at most about two and a half rounds of them (two to
  // an SM); longer calls are bound by bandwidth, which the persistent quantiser uses better.  Whole
  // call, with the short form / without, us: 48 heads of 288 tokens 19.8 / 25.3 (288 CTAs), 1 024
  // tokens 58.2 / 62.3 (576), 1 100 tokens 63.3 / 69.1 (648), 1 536 tokens 100 / 95 (864), 2 048
  // tokens 169 / 154 (1 152); 8 heads of 2 048 tokens 50.4 / 56.4 (192); 40 heads, 8 192 queries of
  // 1 024 keys 236 / 231 (1 600).
  int most_ctas = 0;
  if (!varlen && tk <= SHORT_CTAS) {
    e = (p.qk_mode == 0) ? short_cluster_limit<T, true>(dev, &most_ctas) : short_cluster_limit<T, false>(dev, &most_ctas);
    if (e != cudaSuccess) return e;
  }
  if (!varlen && tk <= most_ctas && bh * tk + (a.BHq * tq + 1) / 2 <= 5 * (int64_t)sm_count[dev]) {
    ShortArgs sa;
    sa.mean = p.mean; sa.vmean = p.vmean; sa.words = words; sa.n_words = (int)CtrlHeader::words(bh); sa.kv_clusters = (int)bh;
    sa.items_q = a.qm ? 0 : a.BHq * tq;      // Q tiles that need K's mean (for the LSE) follow in a launch of their own
    sa.counter_word = (int)CtrlHeader::status_word(bh) + 2;
    sa.items = (unsigned)(2 * bh * tk + sa.items_q);
    e = (p.qk_mode == 0) ? launch_short<T, true>(mq, mk, mv, a, sa, tk, st) : launch_short<T, false>(mq, mk, mv, a, sa, tk, st);
    if (e != cudaSuccess || sa.items_q > 0) return e;
    a.only_q = 1; a.drawn = sa.items;
  } else {
    if (p.plan)
      e = launch_after_predecessor(plan_packed_kernel, dim3(1), dim3(PLAN_MAX_SEQS), 0, st, words, (int)CtrlHeader::words(bh),
                                   p.plan, (int)p.B, p.cu_q, p.cu_k, (long long)p.Tq, (long long)p.Tk, (long long)p.Nq,
                                   (long long)p.N);
    else
      e = launch_after_predecessor(clear_ctrl_kernel, dim3(1), dim3(256), 0, st, words, (int)CtrlHeader::words(bh));
    if (e != cudaSuccess) return e;
    int nsplit = std::min(kmean_splits(bh, p.N, sm_count[dev]), kmean_splits_max(bh, p.N));
    // A packed batch: chunks of 1 024 tokens whatever the number of heads, since its longest sequence
    // would otherwise keep single CTAs busy long after the others (36 k tokens x 48 heads in eleven
    // sequences of up to 8 192: 262 us with one CTA per sequence and head).  CTAs past a sequence's end leave.
    if (p.partial && p.cu_k) {
      const int64_t want = std::min<int64_t>((p.N + 1023) / 1024, (int64_t)(p.partial_bytes / ((size_t)bh * HD * sizeof(double))));
      if (want > nsplit) { nsplit = (int)std::min<int64_t>(want, 65535); partial = reinterpret_cast<double*>(p.partial); }
    }
    long long chunk = (p.N + nsplit - 1) / nsplit;
    chunk = (chunk + 15) / 16 * 16;
    const MeanOf<T> of_k = {reinterpret_cast<const T*>(p.k), p.mean, partial, words, p.k_strides[0], p.k_strides[1], p.k_strides[2]};
    MeanOf<T> of_v = {reinterpret_cast<const T*>(p.v), p.vmean, partial, words + 3 * bh, p.v_strides[0], p.v_strides[1], p.v_strides[2]};
    auto mean_of = [&](const MeanOf<T>& first, const MeanOf<T>& second, unsigned tensors) {
      return launch_after_predecessor(p.cu_k ? kmean_kernel<T, true> : kmean_kernel<T, false>, dim3(nsplit, (unsigned)bh, tensors),
                                      dim3(256), 0, st, first, second, (long long)p.N, (long long)p.H, nsplit, chunk, (int)p.D,
                                      p.cu_k, (long long)p.Tk);
    };
    // V's partial sums go where the staged V factors will be written, if they fit there
    if (p.smooth_k && p.vmean && (size_t)nsplit * HD * sizeof(double) <= (size_t)p.N_pad * sizeof(float)) {
      of_v.partial = reinterpret_cast<double*>(p.svp);
      e = mean_of(of_k, of_v, 2);
    } else {
      if (p.smooth_k) e = mean_of(of_k, of_k, 1);
      if (e == cudaSuccess && p.vmean) e = mean_of(of_v, of_v, 1);
    }
    if (e != cudaSuccess) return e;
  }
  const long long total = (a.only_q ? 0 : 2 * (long long)bh * tk) + (long long)a.BHq * tq;
  long long ctas = (long long)sm_count[dev] * QT_MINBLOCKS;
  if (ctas > total) ctas = total;
  auto kern = varlen ? ((p.qk_mode == 0) ? quant_qkv_kernel<T, true, true> : quant_qkv_kernel<T, false, true>)
                     : ((p.qk_mode == 0) ? quant_qkv_kernel<T, true, false> : quant_qkv_kernel<T, false, false>);
  const int which_kern = (p.qk_mode == 0 ? 1 : 0) | (varlen ? 2 : 0);
  if (!opted_in[dev][which_kern]) {
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)QT_SMEM_BYTES);
    if (e != cudaSuccess) return e;
    opted_in[dev][which_kern] = true;
  }
  return launch_after_predecessor(kern, dim3((unsigned)ctas), dim3(256), QT_SMEM_BYTES, st, mq, mk, mv, a);
}

cudaError_t launch_prologue(const PrologueParams& p, cudaStream_t st) {
  return p.dtype == 0 ? launch_typed<__half>(p, st) : launch_typed<__nv_bfloat16>(p, st);
}

size_t prologue_ctrl_bytes(int64_t B, int64_t H, int64_t N) {
  const int64_t bh = B * H;
  return CtrlHeader::partial_off(bh) + (size_t)bh * kmean_splits_max(bh, N) * HD * sizeof(double);
}

}  // namespace sage
