// KV-cache compaction scores of ScaleKV (models/scalekv/scale_kv.py:232-301) and the row gather that
// builds the compacted cache (pool and gather are byte movers; the scores are bound by latency, see below):
//   scalekv_scores  score[b,h,j] = sum over the window queries i of bf16(bf16(q_i . k_j) / sqrt(D)), -inf on
//                   the window's own columns (the reference's matmul, division, masked_fill and sum on bf16
//                   tensors, rounding where torch rounds); K is read once
//   scalekv_pool    max- or average-pool over `ksize` neighbours (stride 1, padding ksize/2 as torch pads),
//                   then the window columns are raised to +inf so that one exact top-k of max_capacity
//                   entries in ascending index order returns sort(window U top-(max_capacity - w) of the rest),
//                   which is the reference's cat + sort
//   gather_rows     dst[b,h,i,:] = src[b,h,idx[b,h,i],:]
#include <math.h>

#include "common.cuh"
#include "ptx.cuh"

namespace lvar {

namespace {

constexpr int kMaxWindow = 64;

__device__ __forceinline__ float bf16_round(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }

// 1 / sqrt(D) as fp32.  A bf16 logit times this constant rounds to the same bf16 value as the quotient by
// sqrt(D), for every bf16 value (checked over all of them by tests/test_scalekv_oracle.py), so the per-logit division
// is a multiplication.
template <int D>
__device__ __forceinline__ constexpr float inv_sqrt_d() { return D == 64 ? 0.125f : 0.08838834764831845f; }

constexpr int kScoreThreads = 64;                // a thread owns two keys
constexpr int kScoreKeys = 2 * kScoreThreads;    // keys per block
constexpr int kQGroup = 8;                       // window queries in flight: four packed pairs

template <int D>
constexpr size_t scores_smem_bytes(int w) {
  return (size_t)kScoreKeys * (D * 2 + 16) + (size_t)((w + kQGroup - 1) / kQGroup) * D * kQGroup * 4;
}

// Bound by latency: of 35 us at 32 heads x 6425 keys x 16 queries (D = 128; kernel alone) the fp32 pipe needs 12 and K from HBM 8,
// and the ten warps that fit an SM do not cover the rest.  The summation order of a logit is part of the result (its bf16
// rounding decides which keys stay), so the products stay on packed fp32 multiply-adds: D/8 partial sums of 8 consecutive elements, each added up
// in ascending order, then a pairwise tree over the partial sums p and p + D/16, p + D/32, ...  A thread owns two
// whole keys and a group of 8 queries, so that one 16-byte shared-memory read of queries feeds four packed
// multiply-adds; the tree is walked in the order that closes its pairs at once (a binary counter), which keeps at most
// log2(D/8) + 1 partial sums per logit alive.  Nothing crosses lanes.  Only four of the D/8 leaves are unrolled: all of
// them together miss the instruction caches (two stalled cycles per issue).  32 heads x 6425 keys x 16 queries, D = 128:
// 38 us; 42 us with every leaf unrolled; 103 us with a key shared by as many lanes as it has 16-byte pieces, which spends
// four shuffles and sixteen lanes' rounding arithmetic on every logit.
template <int D>
__global__ void __launch_bounds__(kScoreThreads, 5)
scalekv_scores_kernel(const __nv_bfloat16* __restrict__ q, const __nv_bfloat16* __restrict__ k,
                      const int32_t* __restrict__ window, float* __restrict__ scores, int H, int Lq, int Lkv,
                      int64_t q_sb, int64_t q_sh, int64_t q_sl, int64_t k_sb, int64_t k_sh, int64_t k_sl, int w,
                      int offset) {
  constexpr int NP = D / 8;             // 16-byte pieces of a row = leaves of the summation tree
  constexpr int LEVELS = D == 128 ? 4 : 3;
  constexpr int ROW = D * 2 + 16;       // bytes of a staged key row: 16-byte reads of neighbouring rows hit all banks
  extern __shared__ __align__(16) uint8_t sh_keys[];
  float* qf = reinterpret_cast<float*>(sh_keys + kScoreKeys * ROW);  // [query group][D][8] fp32, zeros past w
  __shared__ int wcol[kMaxWindow];
  const int bh = blockIdx.y, b = bh / H, h = bh % H;
  const __nv_bfloat16* qb = q + b * q_sb + h * q_sh;
  const __nv_bfloat16* kb = k + b * k_sb + h * k_sh;
  const int j0 = blockIdx.x * kScoreKeys;
  for (int t = threadIdx.x; t < kScoreKeys * NP; t += kScoreThreads) {
    const int r = t / NP, c = t % NP;
    const int j = min(j0 + r, Lkv - 1);
    cp_async_16(smem_u32(sh_keys + r * ROW + c * 16), kb + (int64_t)j * k_sl + c * 8);
  }
  cp_async_commit();
  // the window queries: query row clamp(window[i] - offset, 0, Lq - 1)
  const int groups = (w + kQGroup - 1) / kQGroup;
  for (int t = threadIdx.x; t < groups * kQGroup * NP; t += kScoreThreads) {
    const int i = t % (groups * kQGroup), c = t / (groups * kQGroup);
    uint4 raw = make_uint4(0, 0, 0, 0);
    if (i < w) {
      const int row = min(max(window[i] - offset, 0), Lq - 1);
      raw = *reinterpret_cast<const uint4*>(qb + (int64_t)row * q_sl + c * 8);
    }
    const uint32_t u[4] = {raw.x, raw.y, raw.z, raw.w};
    float* dst = qf + ((i / kQGroup) * D + c * 8) * kQGroup + i % kQGroup;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      dst[(2 * e) * kQGroup] = __uint_as_float(u[e] << 16);
      dst[(2 * e + 1) * kQGroup] = __uint_as_float(u[e] & 0xffff0000u);
    }
  }
  if (threadIdx.x < w) wcol[threadIdx.x] = window[threadIdx.x];
  cp_async_wait<0>();
  __syncthreads();

  float total[2] = {0.f, 0.f};
  for (int g = 0; g < groups; ++g) {
    uint64_t node[2][4], pair[2][4], hold[2][4], left[2][4];  // [key][query pair]; node: the subtree just closed
#pragma unroll 1
    for (int m = 0; m < NP / 4; ++m) {
      // leaf n of the walk is the piece whose number is n with its bits reversed; leaves 4m .. 4m + 3 close a subtree of
      // four (unrolled), the subtrees close in the same manner in the outer loop
      const int mrev = LEVELS == 4 ? ((m & 1) << 1) | (m >> 1) : m;
      uint64_t first[2][4];
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        const int piece = (((n & 1) << 1 | n >> 1) << (LEVELS - 2)) | mrev;
        asm volatile("" ::: "memory");  // a piece's shared-memory reads stay with it: hoisted, they would spill
        uint64_t acc[2][4];
#pragma unroll
        for (int x = 0; x < 2; ++x)
#pragma unroll
          for (int y = 0; y < 4; ++y) acc[x][y] = 0ull;
        uint32_t ku[2][4];
#pragma unroll
        for (int x = 0; x < 2; ++x) {
          const uint4 raw = *reinterpret_cast<const uint4*>(sh_keys + (threadIdx.x + x * kScoreThreads) * ROW + piece * 16);
          ku[x][0] = raw.x; ku[x][1] = raw.y; ku[x][2] = raw.z; ku[x][3] = raw.w;
        }
        const ulonglong2* qp = reinterpret_cast<const ulonglong2*>(qf + (g * D + piece * 8) * kQGroup);
#pragma unroll
        for (int d = 0; d < 8; ++d) {
          const ulonglong2 qa = qp[2 * d], qc = qp[2 * d + 1];
#pragma unroll
          for (int x = 0; x < 2; ++x) {
            const uint32_t u = ku[x][d >> 1];
            const float kv = __uint_as_float((d & 1) ? (u & 0xffff0000u) : (u << 16));
            const uint64_t kk = pack_f32x2(kv, kv);
            acc[x][0] = ffma2(qa.x, kk, acc[x][0]);
            acc[x][1] = ffma2(qa.y, kk, acc[x][1]);
            acc[x][2] = ffma2(qc.x, kk, acc[x][2]);
            acc[x][3] = ffma2(qc.y, kk, acc[x][3]);
          }
        }
#pragma unroll
        for (int x = 0; x < 2; ++x)
#pragma unroll
          for (int y = 0; y < 4; ++y) {
            if (n == 0 || n == 2) first[x][y] = acc[x][y];
            else if (n == 1) pair[x][y] = fadd2(first[x][y], acc[x][y]);
            else node[x][y] = fadd2(pair[x][y], fadd2(first[x][y], acc[x][y]));
          }
      }
#pragma unroll
      for (int x = 0; x < 2; ++x)
#pragma unroll
        for (int y = 0; y < 4; ++y) {
          if (m & 1) node[x][y] = fadd2(hold[x][y], node[x][y]);
          else hold[x][y] = node[x][y];
          if (LEVELS == 4) {
            if (m == 1) left[x][y] = node[x][y];
            if (m == 3) node[x][y] = fadd2(left[x][y], node[x][y]);
          }
        }
    }
    // the closed tree: logit rounded to bf16 (matmul output), divided by sqrt(D) and rounded again (bf16 / scalar)
#pragma unroll
    for (int x = 0; x < 2; ++x)
#pragma unroll
      for (int y = 0; y < 4; ++y) {
        float lo, hi;
        unpack_f32x2(node[x][y], lo, hi);
        if (g * kQGroup + 2 * y < w) total[x] += bf16_round(bf16_round(lo) * inv_sqrt_d<D>());
        if (g * kQGroup + 2 * y + 1 < w) total[x] += bf16_round(bf16_round(hi) * inv_sqrt_d<D>());
      }
  }
#pragma unroll
  for (int x = 0; x < 2; ++x) {
    const int j = j0 + threadIdx.x + x * kScoreThreads;
    if (j >= Lkv) continue;
    bool in_window = false;
    for (int i = 0; i < w; ++i) in_window |= (wcol[i] == j);
    scores[(int64_t)bh * Lkv + j] = in_window ? -INFINITY : bf16_round(total[x]);
  }
}

// The same logits, sums and bits for few keys: a key is shared by as many lanes as it has 16-byte pieces, so that sixteen
// times as many warps work on it, and a query slot that the window does not fill costs nothing.  Bound by latency like any
// small launch; per key and query it needs three times the instructions of the kernel above (see launch_scalekv_scores).
template <int D>
__global__ void __launch_bounds__(256)
scalekv_scores_few_kernel(const __nv_bfloat16* __restrict__ q, const __nv_bfloat16* __restrict__ k,
                          const int32_t* __restrict__ window, float* __restrict__ scores, int H, int Lq, int Lkv,
                          int64_t q_sb, int64_t q_sh, int64_t q_sl, int64_t k_sb, int64_t k_sh, int64_t k_sl, int w,
                          int offset) {
  constexpr int LPK = D / 8;        // lanes per key
  constexpr int KPB = 8 * 32 / LPK; // keys per block
  __shared__ __align__(16) __nv_bfloat16 wq[kMaxWindow * D];
  __shared__ int wcol[kMaxWindow];
  const int bh = blockIdx.y, b = bh / H, h = bh % H;
  const __nv_bfloat16* qb = q + b * q_sb + h * q_sh;
  const __nv_bfloat16* kb = k + b * k_sb + h * k_sh;
  for (int t = threadIdx.x; t < w * LPK; t += 256) {
    const int i = t / LPK, c = t % LPK;
    const int row = min(max(window[i] - offset, 0), Lq - 1);
    reinterpret_cast<uint4*>(wq)[i * LPK + c] = *reinterpret_cast<const uint4*>(qb + (int64_t)row * q_sl + c * 8);
  }
  if (threadIdx.x < w) wcol[threadIdx.x] = window[threadIdx.x];
  __syncthreads();
  const int piece = threadIdx.x % LPK;
  const int j = blockIdx.x * KPB + threadIdx.x / LPK;
  float kf[8];
  const uint4 kraw = j < Lkv ? *reinterpret_cast<const uint4*>(kb + (int64_t)j * k_sl + piece * 8) : make_uint4(0, 0, 0, 0);
  const uint32_t ku[4] = {kraw.x, kraw.y, kraw.z, kraw.w};
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    kf[2 * e] = __uint_as_float(ku[e] << 16);
    kf[2 * e + 1] = __uint_as_float(ku[e] & 0xffff0000u);
  }
  float total = 0.f;
  for (int i = 0; i < w; ++i) {
    const uint4 raw = reinterpret_cast<const uint4*>(wq)[i * LPK + piece];
    const uint32_t u[4] = {raw.x, raw.y, raw.z, raw.w};
    float dot = 0.f;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      dot = fmaf(__uint_as_float(u[e] << 16), kf[2 * e], dot);
      dot = fmaf(__uint_as_float(u[e] & 0xffff0000u), kf[2 * e + 1], dot);
    }
#pragma unroll
    for (int d = LPK / 2; d >= 1; d >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, d);
    total += bf16_round(bf16_round(dot) * inv_sqrt_d<D>());
  }
  if (piece == 0 && j < Lkv) {
    bool in_window = false;
    for (int i = 0; i < w; ++i) in_window |= (wcol[i] == j);
    scores[(int64_t)bh * Lkv + j] = in_window ? -INFINITY : bf16_round(total);
  }
}

// pooled[j] over neighbours j - r .. j + r (r = ksize / 2); max: torch pads with -inf; average: torch pads
// with zeros and divides by ksize, result rounded to bf16 like the input dtype.  Window columns -> +inf.
__global__ void scalekv_pool_kernel(const float* __restrict__ scores, const int32_t* __restrict__ window, int w,
                                    float* __restrict__ pooled, int Lkv, int ksize, int avg) {
  __shared__ int wcol[kMaxWindow];
  if (threadIdx.x < w) wcol[threadIdx.x] = window[threadIdx.x];
  __syncthreads();
  const int64_t row = blockIdx.y;
  const float* s = scores + row * Lkv;
  const int r = ksize / 2;
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < Lkv; j += gridDim.x * blockDim.x) {
    float acc = avg ? 0.f : -INFINITY;
    for (int d = -r; d <= r; ++d) {
      const int t = j + d;
      if (t < 0 || t >= Lkv) continue;
      acc = avg ? acc + s[t] : fmaxf(acc, s[t]);
    }
    if (avg) acc = bf16_round(acc / (float)ksize);
    bool in_window = false;
    for (int i = 0; i < w; ++i) in_window |= (wcol[i] == j);
    pooled[row * Lkv + j] = in_window ? INFINITY : acc;
  }
}

// Bound by HBM once the index arithmetic is out of the way: D/8 threads copy a row in 16-byte pieces, a thread keeps its
// piece number and walks rows (four in flight), a (batch, head) per grid row.  2000 of 6425 rows of 256 bytes, 32 heads:
// 5.8 us; 7.7 us with 64-bit divisions and remainders for every piece.
constexpr int kGatherThreads = 256;
template <int ROWS>
__global__ void __launch_bounds__(kGatherThreads)
gather_rows_kernel(const __nv_bfloat16* __restrict__ src, const int32_t* __restrict__ idx, __nv_bfloat16* __restrict__ dst,
                   int H, int L, int n, int D, int64_t s_sb, int64_t s_sh, int64_t s_sl, int64_t idx_row_stride, int BH) {
  const int ppr = D / 8;  // pieces per row
  const int rpb = max(1, kGatherThreads / ppr);
  const int r = (int)threadIdx.x / ppr;
  if (r >= rpb) return;
  const int c0 = (int)threadIdx.x - r * ppr;
  for (int bh = blockIdx.y; bh < BH; bh += gridDim.y) {
    const int b = bh / H, h = bh - b * H;
    const __nv_bfloat16* s = src + b * s_sb + h * s_sh;
    const int32_t* ix = idx + bh * idx_row_stride;
    uint4* d = reinterpret_cast<uint4*>(dst) + (int64_t)bh * n * ppr;
    for (int64_t i0 = (int64_t)blockIdx.x * rpb * ROWS + r; i0 < n; i0 += (int64_t)gridDim.x * rpb * ROWS) {
      int row[ROWS];
#pragma unroll
      for (int u = 0; u < ROWS; ++u) {
        const int64_t i = i0 + u * rpb;
        row[u] = i < n ? min(max(ix[i], 0), L - 1) : 0;
      }
      for (int c = c0; c < ppr; c += kGatherThreads) {  // more than one pass only for rows above 4 KB
        uint4 v[ROWS];
#pragma unroll
        for (int u = 0; u < ROWS; ++u) v[u] = *reinterpret_cast<const uint4*>(s + row[u] * s_sl + c * 8);
#pragma unroll
        for (int u = 0; u < ROWS; ++u) {
          const int64_t i = i0 + u * rpb;
          if (i < n) d[i * ppr + c] = v[u];
        }
      }
    }
  }
}

}  // namespace

int launch_scalekv_scores(const void* q, const void* k, const int32_t* window, float* scores, int B, int H, int Lq,
                          int Lkv, int D, int64_t q_sb, int64_t q_sh, int64_t q_sl, int64_t k_sb, int64_t k_sh,
                          int64_t k_sl, int w, int offset, cudaStream_t stream) {
  LVAR_REQUIRE(q && k && window && scores, LVAR_ERR_ARG, "q, k, window and scores must be non-null");
  LVAR_REQUIRE(D == 64 || D == 128, LVAR_ERR_UNSUPPORTED, "Head dimension must be 64 or 128 (got %d)", D);
  LVAR_REQUIRE(B >= 1 && H >= 1 && Lq >= 1 && Lkv >= 1, LVAR_ERR_ARG, "B, H, Lq, Lkv must be >= 1");
  LVAR_REQUIRE(w >= 1 && w <= kMaxWindow, LVAR_ERR_UNSUPPORTED, "window of %d queries (supported: 1..%d)", w, kMaxWindow);
  LVAR_REQUIRE(aligned16(q) && aligned16(k), LVAR_ERR_ARG, "q and k must be 16-byte aligned");
  const int64_t strides[] = {q_sb, q_sh, q_sl, k_sb, k_sh, k_sl};
  for (int64_t s : strides)
    LVAR_REQUIRE(s % 8 == 0 && s >= 0, LVAR_ERR_ARG, "tensor strides must be non-negative multiples of 8 elements");
  LVAR_REQUIRE((int64_t)B * H <= 65535, LVAR_ERR_UNSUPPORTED, "B*H must be <= 65535");
  // Few keys: the launch takes as long as one block, and a block of whole keys per thread pays 5.6 us plus 3 us per further
  // group of eight queries (4.2 and 1.5 us with D = 64) where shared keys pay 2.2 us plus 0.28 us per query.  The lines
  // are where the measured times cross, in keys times the used share of the query slots (one head of 200 keys, 16 queries:
  // 5.9 against 8.3 us; 16 heads of 680 keys, one query, D = 64: 2.6 against 4.1 us; 32 heads of 265 keys, 16 queries: 8.8
  // both ways).
  const int slots = (w + kQGroup - 1) / kQGroup * kQGroup;
  const bool few = (int64_t)B * H * Lkv * w < 9000ll * slots && (D == 128 || 4 * w <= 3 * slots);
  const int kpb = few ? 8 * 32 / (D / 8) : kScoreKeys;
  dim3 grid((unsigned)((Lkv + kpb - 1) / kpb), (unsigned)(B * H));
  const auto* qp = static_cast<const __nv_bfloat16*>(q);
  const auto* kp = static_cast<const __nv_bfloat16*>(k);
  const size_t smem = D == 128 ? scores_smem_bytes<128>(w) : scores_smem_bytes<64>(w);
  if (few) {
    auto kern = D == 128 ? scalekv_scores_few_kernel<128> : scalekv_scores_few_kernel<64>;
    kern<<<grid, 256, 0, stream>>>(qp, kp, window, scores, H, Lq, Lkv, q_sb, q_sh, q_sl, k_sb, k_sh, k_sl, w, offset);
  } else if (D == 128) {
    LVAR_CUDA_OK(cudaFuncSetAttribute(scalekv_scores_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)scores_smem_bytes<128>(kMaxWindow)));
    scalekv_scores_kernel<128><<<grid, kScoreThreads, smem, stream>>>(qp, kp, window, scores, H, Lq, Lkv, q_sb, q_sh, q_sl,
                                                                      k_sb, k_sh, k_sl, w, offset);
  } else {
    scalekv_scores_kernel<64><<<grid, kScoreThreads, smem, stream>>>(qp, kp, window, scores, H, Lq, Lkv, q_sb, q_sh, q_sl,
                                                                     k_sb, k_sh, k_sl, w, offset);
  }
  LVAR_CUDA_OK(cudaGetLastError());
  return LVAR_OK;
}

int launch_scalekv_pool(const float* scores, const int32_t* window, int w, float* pooled, int64_t rows, int Lkv,
                        int ksize, int avg, cudaStream_t stream) {
  LVAR_REQUIRE(scores && window && pooled, LVAR_ERR_ARG, "scores, window and pooled must be non-null");
  LVAR_REQUIRE(rows >= 1 && rows <= 65535 && Lkv >= 1, LVAR_ERR_ARG, "bad sizes");
  LVAR_REQUIRE(w >= 1 && w <= kMaxWindow, LVAR_ERR_UNSUPPORTED, "window of %d queries (supported: 1..%d)", w, kMaxWindow);
  LVAR_REQUIRE(ksize >= 1 && (ksize & 1), LVAR_ERR_ARG, "pooling kernel size must be odd and >= 1 (got %d)", ksize);
  int bx = (Lkv + 255) / 256;
  if (bx > 64) bx = 64;
  scalekv_pool_kernel<<<dim3((unsigned)bx, (unsigned)rows), 256, 0, stream>>>(scores, window, w, pooled, Lkv, ksize, avg);
  LVAR_CUDA_OK(cudaGetLastError());
  return LVAR_OK;
}

int launch_gather_rows(const void* src, const int32_t* idx, void* dst, int B, int H, int L, int n, int D, int64_t s_sb,
                       int64_t s_sh, int64_t s_sl, int64_t idx_row_stride, cudaStream_t stream) {
  LVAR_REQUIRE(src && idx && dst, LVAR_ERR_ARG, "src, idx and dst must be non-null");
  LVAR_REQUIRE(B >= 1 && H >= 1 && L >= 1 && n >= 1, LVAR_ERR_ARG, "B, H, L, n must be >= 1");
  LVAR_REQUIRE(D >= 8 && D % 8 == 0, LVAR_ERR_ARG, "row length must be a positive multiple of 8 elements (got %d)", D);
  LVAR_REQUIRE(aligned16(src) && aligned16(dst), LVAR_ERR_ARG, "src and dst must be 16-byte aligned");
  LVAR_REQUIRE(s_sb % 8 == 0 && s_sh % 8 == 0 && s_sl % 8 == 0, LVAR_ERR_ARG,
               "tensor strides must be multiples of 8 elements");
  LVAR_REQUIRE(idx_row_stride >= n, LVAR_ERR_ARG, "index rows shorter than n");
  LVAR_REQUIRE((int64_t)B * H < (1ll << 31), LVAR_ERR_LIMIT, "too many rows");
  const int bh = B * H, rpb = D / 8 < kGatherThreads ? kGatherThreads / (D / 8) : 1;
  // four rows per thread once that still gives every SM two blocks; below, one row each
  const int64_t bx4 = ((int64_t)n + (int64_t)rpb * 4 - 1) / ((int64_t)rpb * 4);
  const bool four = bx4 * bh >= 2 * 148;
  const int64_t bx = four ? bx4 : ((int64_t)n + rpb - 1) / rpb;
  const dim3 grid((unsigned)(bx < (1ll << 30) ? bx : (1ll << 30)), (unsigned)(bh < 65535 ? bh : 65535));
  auto kern = four ? gather_rows_kernel<4> : gather_rows_kernel<1>;
  kern<<<grid, kGatherThreads, 0, stream>>>(static_cast<const __nv_bfloat16*>(src), idx, static_cast<__nv_bfloat16*>(dst), H,
                                            L, n, D, s_sb, s_sh, s_sl, idx_row_stride, bh);
  LVAR_CUDA_OK(cudaGetLastError());
  return LVAR_OK;
}

}  // namespace lvar
