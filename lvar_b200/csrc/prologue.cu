// QKV prologue of a self-attention layer during generation (models/sparvar/basic_sparvar.py:321-350,
// models/infinity/basic_infinity.py:111-133), one HBM-bound pass instead of normalize, mul, stack, RoPE,
// two torch.cat of the whole KV cache and a cast of the cache at every attention call:
//   q_out[b,h,l,:]            = bf16( rope( q / max(|q|, 1e-12) * scale_mul[h] ) )
//   k_cache[b,h,pos + l,:]    = bf16( rope( k / max(|k|, 1e-12) ) )
//   v_cache[b,h,pos + l,:]    = v
// from the projection output qkv bf16 [B, L, 3, H, c].  All arithmetic in fp32 on the widened bf16 inputs,
// in the reference's order (division by the clamped norm, then the per-head scale, then the rotation with
// separate multiplies and add/subtract), one rounding to bf16 at the end: the reference keeps q and k in
// fp32 and casts them to v's dtype at every call site.
// rope(x)[2i] = cos[p,i] x[2i] - sin[p,i] x[2i+1],  rope(x)[2i+1] = sin[p,i] x[2i] + cos[p,i] x[2i+1],
// p = rope_start + l.
//
// Bound by HBM (12 c bytes per token and head, every byte once) as long as the arithmetic stays below it: c / 8 lanes
// share a (b, l, h) row and hold 8 consecutive elements each (16-byte accesses), a warp takes one token and a few heads
// so that the rotation table is read once for all of them, and every index is 32-bit.  A warp per row with 4 or 2
// elements per lane, 64-bit index divisions and a library division per element was bound by instruction issue:
// 66 us for 2 x 4096 tokens x 16 heads x 128 and 256 us for 8 x 4096, now 36 and 135 us (6.0 TB/s).
#include <math.h>

#include "common.cuh"
#include "ptx.cuh"

namespace lvar {

namespace {

struct PrologueParams {
  const __nv_bfloat16* qkv;
  int64_t s_b, s_l, s_w, s_h;
  const float* scale_mul;  // [H] or nullptr (no normalisation at all: plain copy + optional RoPE)
  const float* cos_t;      // [*, c/2] or nullptr (no RoPE)
  const float* sin_t;
  int rope_start;
  __nv_bfloat16* q_out;
  int64_t q_sb, q_sh, q_sl;
  __nv_bfloat16* k_cache;
  int64_t k_sb, k_sh, k_sl;
  __nv_bfloat16* v_cache;
  int64_t v_sb, v_sh, v_sl;
  int cache_pos;
  int B, L, H;
};

// a / b rounded to nearest, for r = 1 / b rounded to nearest: the residual of the first quotient is exact in a fused
// multiply-add and corrects it (Markstein, "Computation of elementary functions on the IBM RISC System/6000
// processor", 1990).  Three instructions per element once the row's reciprocal is known.  Exact while the quotient is a
// normal number and the residual does not fall below the subnormal step: for b in [1e-12, 2^64], a zero or |a| >= 2^-62.
// The residual is formed with its sign reversed, so that a zero keeps its own.
__device__ __forceinline__ float div_by(float a, float b, float r) {
  const float q = __fmul_rn(a, r);
  return fmaf(-fmaf(q, b, -a), r, q);
}

// Whether all eight bf16 elements are ones that div_by takes, where some are zeros or tiny.  Per 16-bit half: magnitude
// + 0x7fff has no carry and, as a signed number, is largest for a zero and ascending for the others; 0x2080 is 2^-62.
__device__ __forceinline__ bool div_by_takes(const uint32_t (&u)[4]) {
  uint32_t least = 0x7fff7fffu;
#pragma unroll
  for (int i = 0; i < 4; ++i) least = __vmins2(least, (u[i] & 0x7fff7fffu) + 0x7fff7fffu);
  constexpr int kTiny = (int)(0xa07fu << 16);
  return (int)(least << 16) >= kTiny && (int)(least & 0xffff0000u) >= kTiny;
}

template <bool WIDE>
__device__ __forceinline__ uint4 load8(const __nv_bfloat16* p) {
  if (WIDE) return *reinterpret_cast<const uint4*>(p);
  const uint2 lo = reinterpret_cast<const uint2*>(p)[0], hi = reinterpret_cast<const uint2*>(p)[1];
  return make_uint4(lo.x, lo.y, hi.x, hi.y);
}
template <bool WIDE>
__device__ __forceinline__ void store8(__nv_bfloat16* p, const uint4& v) {
  if (WIDE) {
    *reinterpret_cast<uint4*>(p) = v;
  } else {
    reinterpret_cast<uint2*>(p)[0] = make_uint2(v.x, v.y);
    reinterpret_cast<uint2*>(p)[1] = make_uint2(v.z, v.w);
  }
}
template <bool WIDE>
__device__ __forceinline__ void load4f(const float* p, float (&out)[4]) {
  if (WIDE) {
    const float4 v = __ldg(reinterpret_cast<const float4*>(p));
    out[0] = v.x; out[1] = v.y; out[2] = v.z; out[3] = v.w;
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i) out[i] = __ldg(p + i);
  }
}

// One warp: ROWS * 32 / (C / 8) rows, all loads issued before any arithmetic.  Its 32 / (C / 8) groups of C / 8 lanes
// take 1 << hsh heads of as many tokens as that leaves (one token but for tensors with one or two heads).  WIDE: every
// base and stride allows 16-byte accesses (else 8-byte ones, and single floats from the tables).
template <int C, bool WIDE, int ROWS>
__global__ void __launch_bounds__(256) qkv_prologue_kernel(const PrologueParams p, int units, int chunks, int hsh) {
  constexpr int LPR = C / 8;        // lanes per row
  constexpr int LOG_RPW = C == 128 ? 1 : 2;  // 32 / LPR rows per warp at a time
  const int lane = threadIdx.x & 31;
  const int unit = (int)blockIdx.x * (int)(blockDim.x >> 5) + (int)(threadIdx.x >> 5);
  if (unit >= units) return;
  const int g = lane / LPR;
  const int sh = ROWS == 2 ? LOG_RPW : hsh;  // two rows per lane: one token per warp
  const int tu = unit / chunks;
  const int t = (tu << (LOG_RPW - sh)) + (g >> sh);  // token over the batch
  const int b = t / p.L, l = t - b * p.L;
  const int hstep = 1 << sh;
  // a lane past the last token takes part in the shuffles without a head
  const int h0 = t < p.B * p.L ? (((unit - tu * chunks) * ROWS) << sh) + (g & (hstep - 1)) : p.H;
  const int e0 = (lane % LPR) * 8;  // this lane's first element
  const __nv_bfloat16* src = p.qkv + b * p.s_b + l * p.s_l + e0;
  uint4 raw[ROWS][3];
#pragma unroll
  for (int r = 0; r < ROWS; ++r) {
    const int h = h0 + r * hstep;
    if (h < p.H) {
#pragma unroll
      for (int which = 0; which < 3; ++which) raw[r][which] = load8<WIDE>(src + h * p.s_h + which * p.s_w);
    } else {
      // ones: nothing that leaves the fast path of the division
      raw[r][0] = raw[r][1] = raw[r][2] = make_uint4(0x3f803f80u, 0x3f803f80u, 0x3f803f80u, 0x3f803f80u);
    }
  }
  float mul[ROWS];
#pragma unroll
  for (int r = 0; r < ROWS; ++r) mul[r] = p.scale_mul != nullptr && h0 + r * hstep < p.H ? p.scale_mul[h0 + r * hstep] : 1.0f;
  float cs[4], sn[4];
  if (p.cos_t != nullptr && h0 < p.H) {
    const int64_t base = (int64_t)(p.rope_start + l) * (C / 2) + (e0 >> 1);
    load4f<WIDE>(p.cos_t + base, cs);
    load4f<WIDE>(p.sin_t + base, sn);
  }
#pragma unroll
  for (int r = 0; r < ROWS; ++r) {
    const int h = h0 + r * hstep;
    const bool live = h < p.H;  // lanes past the last head still take part in the shuffles
    uint4 out[2];
#pragma unroll
    for (int which = 0; which < 2; ++which) {
      const uint32_t u[4] = {raw[r][which].x, raw[r][which].y, raw[r][which].z, raw[r][which].w};
      float x[8];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        x[2 * i] = __uint_as_float(u[i] << 16);
        x[2 * i + 1] = __uint_as_float(u[i] & 0xffff0000u);
      }
      if (p.scale_mul != nullptr) {
        // squares of EPS consecutive elements are summed in order, then a pairwise tree over the row's 32 such sums
        constexpr int EPS = C / 32;
        constexpr int NS = 8 / EPS;  // sums this lane starts with
        float ssq[NS];
#pragma unroll
        for (int i = 0; i < NS; ++i) {
          ssq[i] = 0.f;
#pragma unroll
          for (int e = 0; e < EPS; ++e) ssq[i] = fmaf(x[i * EPS + e], x[i * EPS + e], ssq[i]);
#pragma unroll
          for (int d = LPR / 2; d >= 1; d >>= 1) ssq[i] += __shfl_xor_sync(0xffffffffu, ssq[i], d);
        }
#pragma unroll
        for (int d = NS / 2; d >= 1; d >>= 1)
#pragma unroll
          for (int i = 0; i < d; ++i) ssq[i] += ssq[i + d];
        const float denom = fmaxf(sqrtf(ssq[0]), 1e-12f);
        float least = fabsf(x[0]);
#pragma unroll
        for (int e = 1; e < 8; ++e) least = fminf(least, fabsf(x[e]));
        if (ssq[0] < INFINITY && (least >= 0x1p-62f || div_by_takes(u))) {
          // denom lies in [1e-12, 2^64] and no quotient overflows
          const float inv = __frcp_rn(denom);
#pragma unroll
          for (int e = 0; e < 8; ++e) x[e] = div_by(x[e], denom, inv);
        } else {  // an infinite or NaN sum of squares, a tiny element
#pragma unroll
          for (int e = 0; e < 8; ++e) x[e] = __fdiv_rn(x[e], denom);
        }
        if (which == 0) {
#pragma unroll
          for (int e = 0; e < 8; ++e) x[e] = __fmul_rn(x[e], mul[r]);
        }
      }
      if (p.cos_t != nullptr) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float a = x[2 * i], b2 = x[2 * i + 1];
          x[2 * i] = __fsub_rn(__fmul_rn(cs[i], a), __fmul_rn(sn[i], b2));
          x[2 * i + 1] = __fadd_rn(__fmul_rn(sn[i], a), __fmul_rn(cs[i], b2));
        }
      }
      out[which] = make_uint4(pack_bf16x2(x[0], x[1]), pack_bf16x2(x[2], x[3]), pack_bf16x2(x[4], x[5]),
                              pack_bf16x2(x[6], x[7]));
    }
    if (live) {
      const int64_t pos = p.cache_pos + l;
      store8<WIDE>(p.q_out + b * p.q_sb + h * p.q_sh + l * p.q_sl + e0, out[0]);
      store8<WIDE>(p.k_cache + b * p.k_sb + h * p.k_sh + pos * p.k_sl + e0, out[1]);
      store8<WIDE>(p.v_cache + b * p.v_sb + h * p.v_sh + pos * p.v_sl + e0, raw[r][2]);
    }
  }
}

template <int C, int ROWS>
int launch_c(const PrologueParams& p, bool wide, cudaStream_t stream) {
  constexpr int LOG_RPW = C == 128 ? 1 : 2;
  int hsh = 0;
  while (hsh < LOG_RPW && (ROWS == 2 || (1 << hsh) < p.H)) ++hsh;
  const int chunks = (p.H + (ROWS << hsh) - 1) / (ROWS << hsh);
  const int64_t tokens = (int64_t)p.B * p.L, per = 1 << (LOG_RPW - hsh);
  const int64_t units = (tokens + per - 1) / per * chunks;
  LVAR_REQUIRE(units < (1ll << 31) - 8 && tokens < (1ll << 31) - 8, LVAR_ERR_LIMIT, "too many rows");
  const unsigned blocks = (unsigned)((units + 7) / 8);
  if (wide) qkv_prologue_kernel<C, true, ROWS><<<blocks, 256, 0, stream>>>(p, (int)units, chunks, hsh);
  else qkv_prologue_kernel<C, false, ROWS><<<blocks, 256, 0, stream>>>(p, (int)units, chunks, hsh);
  LVAR_CUDA_OK(cudaGetLastError());
  return LVAR_OK;
}

// Two rows per lane once one row each would fill the chip twice over and the heads pad to the same number either way
// (without normalisation, which is bound by memory alone, to at most a third more): 2 x 4096 x 16 x 128 36 against 41 us
// with one.  One row otherwise: half the chain of dependent steps, which is all that a small call waits for (2 x 64 x 16 x
// 128 2.8 against 3.8 us), and no idle lanes (2 x 4096 x 2 x 128 6.1 against 8.3, x 9 heads x 64 14.5 against 16.0).
template <int C>
int launch_rows(const PrologueParams& p, bool wide, cudaStream_t stream) {
  constexpr int LOG_RPW = C == 128 ? 1 : 2;
  const int64_t step = p.H > 1 << (LOG_RPW - 1) ? 1 << LOG_RPW : p.H;  // heads per warp with one row per lane
  const int64_t chunks = (p.H + step - 1) / step, even = (chunks + 1) / 2 * 2;
  const int64_t units = (int64_t)p.B * p.L * chunks;
  const bool fits = even == chunks || (p.scale_mul == nullptr && 3 * even <= 4 * chunks);
  return fits && units >= 2 * 148 * 40 ? launch_c<C, 2>(p, wide, stream) : launch_c<C, 1>(p, wide, stream);
}

}  // namespace

int launch_qkv_prologue(const void* qkv, int64_t s_b, int64_t s_l, int64_t s_w, int64_t s_h, const float* scale_mul,
                        const float* rope_cos, const float* rope_sin, int rope_start, void* q_out, int64_t q_sb,
                        int64_t q_sh, int64_t q_sl, void* k_cache, int64_t k_sb, int64_t k_sh, int64_t k_sl,
                        void* v_cache, int64_t v_sb, int64_t v_sh, int64_t v_sl, int cache_pos, int B, int L, int H,
                        int c, cudaStream_t stream) {
  LVAR_REQUIRE(qkv && q_out && k_cache && v_cache, LVAR_ERR_ARG, "qkv, q_out, k_cache and v_cache must be non-null");
  LVAR_REQUIRE(c == 64 || c == 128, LVAR_ERR_UNSUPPORTED, "Head dimension must be 64 or 128 (got %d)", c);
  LVAR_REQUIRE(B >= 1 && L >= 1 && H >= 1 && cache_pos >= 0 && rope_start >= 0, LVAR_ERR_ARG, "bad sizes");
  LVAR_REQUIRE((rope_cos == nullptr) == (rope_sin == nullptr), LVAR_ERR_ARG, "rope_cos and rope_sin go together");
  const int64_t strides[] = {s_b, s_l, s_w, s_h, q_sb, q_sh, q_sl, k_sb, k_sh, k_sl, v_sb, v_sh, v_sl};
  for (int64_t s : strides) LVAR_REQUIRE(s % 4 == 0 && s >= 0, LVAR_ERR_ARG, "strides must be non-negative multiples of 4 elements");
  const uintptr_t ptrs[] = {(uintptr_t)qkv, (uintptr_t)q_out, (uintptr_t)k_cache, (uintptr_t)v_cache};
  for (uintptr_t a : ptrs) LVAR_REQUIRE(a % 8 == 0, LVAR_ERR_ARG, "tensors must be 8-byte aligned");
  PrologueParams p{};
  p.qkv = static_cast<const __nv_bfloat16*>(qkv);
  p.s_b = s_b; p.s_l = s_l; p.s_w = s_w; p.s_h = s_h;
  p.scale_mul = scale_mul;
  p.cos_t = rope_cos; p.sin_t = rope_sin; p.rope_start = rope_start;
  p.q_out = static_cast<__nv_bfloat16*>(q_out); p.q_sb = q_sb; p.q_sh = q_sh; p.q_sl = q_sl;
  p.k_cache = static_cast<__nv_bfloat16*>(k_cache); p.k_sb = k_sb; p.k_sh = k_sh; p.k_sl = k_sl;
  p.v_cache = static_cast<__nv_bfloat16*>(v_cache); p.v_sb = v_sb; p.v_sh = v_sh; p.v_sl = v_sl;
  p.cache_pos = cache_pos;
  p.B = B; p.L = L; p.H = H;
  // 16-byte accesses where every row starts on a 16-byte boundary; 8-byte ones otherwise
  bool wide = (uintptr_t)rope_cos % 16 == 0 && (uintptr_t)rope_sin % 16 == 0;
  for (int64_t s : strides) wide = wide && s % 8 == 0;
  for (uintptr_t a : ptrs) wide = wide && a % 16 == 0;
  return c == 128 ? launch_rows<128>(p, wide, stream) : launch_rows<64>(p, wide, stream);
}

}  // namespace lvar
