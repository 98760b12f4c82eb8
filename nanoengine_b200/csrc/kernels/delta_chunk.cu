// Gated delta rule over long portions, chunk by chunk (64 tokens) with matrix instructions, in 32-bit accuracy; 128 x 128 states.
//     S_t = e^(g_t) S_(t-1) (I - b_t k_t k_t^T) + b_t v_t k_t^T,   o_t = S_t q_t
// Inside a chunk with G_t = g_1 + .. + g_t the writes u_t solve a unit lower triangular system,
//     (I + A) U = b (V - e^G K S_0^T),  A_ti = b_t e^(G_t - G_i) k_t.k_i (i < t),     T = (I + A)^-1
//     O = e^G Q S_0^T + P U,            P_ti = e^(G_t - G_i) q_t.k_i (i <= t)
//     S = e^(G_C) S_0 + (e^(G_C - G) U)^T K
// (q, k: unit vectors, q scaled.)  Two kernels:
//   prepare  everything that does not need the state, all chunks at once: T and P T (so that U and the inside part of O come from one product), and the
//            factors of every row.  K K^T and Q K^T on the tensor cores from the bf16 rows as they are, norms as factors behind the product; the inverse by
//            blocks of 16, 32, 64 in fp32.
//   scan     one CTA per (sequence, head, 32 of the 128 value columns - columns are independent of each other given T and P T -) walks the chunks with its
//            part of the state in registers.  Four short products in a row per chunk, 32 x 128 x 128 and smaller, each waiting for the one before.
// A 32-bit operand enters a product as three bf16 terms (x = h + m + l to 2^-25); k and q are bf16 already and enter once, so K S^T and U^T K take three
// products, T R and P T R six.
// Warp-level mma.sync and not tcgen05: S, R and U change between accumulator and operand three times a chunk, which here is a pack in registers (the
// accumulator of a transposed product has the layout of the next product's A operand) and one exchange through shared memory, without the trip through
// TMEM, the descriptor tiles and a commit for each.
// Sums of log decays are 64-bit (64 numbers a chunk): a factor between two tokens is the exponential of a difference of sums.  The tensor cores cut off
// what falls below an accumulator's last bit, so the state is not an accumulator of theirs: a chunk's products are summed from zero and then added.
//
// Bound: the scan's chain of four products a chunk, two CTAs per SM: tensor pipe 49 % busy, shared memory and barriers between the products the rest; in the
// preparation the barriers between its steps (issue slots 51 % busy).  Measured: 4 prompts of 750 .. 2250 tokens, 32 heads over 16: 14774 us as batched fp32 products and triangular
// solves of a library per sequence, 571 us so (under a profiler: prepare 172, scan 371, norm 55).  Errors against 64 bits: final states 1.8e-7 (before: 1.8e-7), outputs in front of the norm 4.3e-7 (3.6e-6 with two
// terms of P T and of R).
//
// Replaces in the reference: the chunked prefill of triton/fla (layers/backends/delta_net/components/recurrence.py:100-200).
#include "ptx.cuh"
#include "seq_tile.cuh"

namespace ne {

[[maybe_unused]] constexpr int kKernelDc = 28;      // in status words of the checked build
constexpr int kDcC = 64;                       // tokens per chunk
constexpr int kDcD = 128;                      // key and value size
constexpr int kDcThreads = 256;
constexpr int kDcPairs = 10;                   // (row block j, column block i <= j) of 16 x 16 of a lower triangular 64 x 64
constexpr int kDcFragBytes = kDcPairs * 2 * 3 * 512;        // T and P T in three terms; 512 bytes: 16 x 16 as the B operands of two mma (16 B per lane)

struct DcArgs {
  const __nv_bfloat16* q; const __nv_bfloat16* k; const __nv_bfloat16* v; long long qk_ld, v_ld;
  const __nv_bfloat16* a; const __nv_bfloat16* b; long long ab_ld;
  const float* A_log; const float* dt_bias;
  float* state; const int* slots; const int* cu; const int* fresh;
  float* raw;                                  // [T, Hv, 128]
  uint8_t* frags; float4* rows; float* decay;  // per (chunk, head): kDcFragBytes, 64 rows of {b, b |k|^-1 e^G, |q|^-1 e^G / sqrt(128), |k|^-1 e^(G_C - G)}, e^(G_C)
  int num_seqs, Hk, Hv, min_n;
};

__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm4t(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
// rows of 128 bf16 (256 bytes), 16-byte pieces permuted so that eight rows of one column are free of bank conflicts
__device__ __forceinline__ uint32_t dc_at(uint32_t base, int row, int piece) { return base + row * 256 + ((piece ^ (row & 7)) << 4); }
// fp32 pair -> three bf16 terms
__device__ __forceinline__ void split3(float a, float b, uint32_t& h, uint32_t& m, uint32_t& l) {
  h = pack_bf16x2(a, b);
  const float2 x = unpack_bf16x2(h);
  a -= x.x; b -= x.y;
  m = pack_bf16x2(a, b);
  const float2 y = unpack_bf16x2(m);
  l = pack_bf16x2(a - y.x, b - y.y);
}
__device__ __forceinline__ uint4 ld_shared_v4(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
  return v;
}

constexpr int kDcLd = 68;                      // row stride of the fp32 64 x 64 matrices

__device__ __forceinline__ int dc_pair(int j, int i) { return j * (j + 1) / 2 + i; }

// rows of q and k of a chunk into shared memory; rows past m are zero
__device__ __forceinline__ void dc_load(uint32_t dst, const __nv_bfloat16* src, long long ld, int m) {
  for (int i = threadIdx.x; i < kDcC * 16; i += kDcThreads) {
    const int r = i >> 4, p = i & 15;
    cp_async16(dc_at(dst, r, p), src + (long long)(r < m ? r : 0) * ld + p * 8, r < m ? 16 : 0);
  }
}

__global__ void __launch_bounds__(kDcThreads, 3) delta_chunk_prepare_kernel(const DcArgs a) {
  pdl_wait(); pdl_trigger();
  extern __shared__ __align__(16) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~uintptr_t(127));
  const uint32_t sK = smem_u32(smem), sQ = sK + kDcC * 256;
  float* sT = reinterpret_cast<float*>(smem);                          // over K and Q, once they have been multiplied
  float* sM = sT + kDcC * kDcLd;                                       // [32][33]
  float* sA = reinterpret_cast<float*>(smem + 2 * kDcC * 256);
  float* sP = sA + kDcC * kDcLd;
  __shared__ double s_g[kDcC];
  __shared__ float s_kn[kDcC], s_qn[kDcC], s_b[kDcC];
  __shared__ int s_seq, s_tok;
  const int h = blockIdx.y, hk = h / (a.Hv / a.Hk), tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (warp == 0) {
    int seq, tok;
    find_seq_tile(a.cu, a.num_seqs, kDcC, blockIdx.x, seq, tok);
    if (lane == 0) { s_seq = seq; s_tok = tok; }
  }
  __syncthreads();
  const int seq = s_seq, t0 = s_tok;
  if (seq < 0) return;
  const int end = a.cu[seq + 1];
  if (end - a.cu[seq] < a.min_n) return;
  const int m = min(kDcC, end - t0);
  dc_load(sK, a.k + (long long)t0 * a.qk_ld + hk * kDcD, a.qk_ld, m);
  dc_load(sQ, a.q + (long long)t0 * a.qk_ld + hk * kDcD, a.qk_ld, m);
  cp_async_commit();
  if (warp == 0) {            // gates, two tokens a lane
    double g[2];
#pragma unroll
    for (int e = 0; e < 2; e++) {
      const int t = lane * 2 + e;
      float y = 0.f, b = 0.f;
      if (t < m) {
        const float x = __bfloat162float(a.a[(long long)(t0 + t) * a.ab_ld + h]) + a.dt_bias[h];
        y = -expf(a.A_log[h]) * (x > 20.f ? x : log1pf(expf(x)));
        b = 1.f / (1.f + expf(-__bfloat162float(a.b[(long long)(t0 + t) * a.ab_ld + h])));
      }
      g[e] = y; s_b[t] = b;
    }
    double sum = g[0] + g[1];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const double x = __shfl_up_sync(0xffffffffu, sum, o); if (lane >= o) sum += x; }
    s_g[lane * 2] = sum - g[1]; s_g[lane * 2 + 1] = sum;
  }
  cp_async_wait<0>();
  __syncthreads();
  {                           // norms: four lanes a row
    const int r = tid >> 2, part = tid & 3;
    float kk = 0.f, qq = 0.f;
#pragma unroll
    for (int p = 0; p < 4; p++) {
      const uint4 uk = ld_shared_v4(dc_at(sK, r, part * 4 + p)), uq = ld_shared_v4(dc_at(sQ, r, part * 4 + p));
      const uint32_t wk[4] = {uk.x, uk.y, uk.z, uk.w}, wq[4] = {uq.x, uq.y, uq.z, uq.w};
#pragma unroll
      for (int e = 0; e < 4; e++) {
        const float2 x = unpack_bf16x2(wk[e]), y = unpack_bf16x2(wq[e]);
        kk = fmaf(x.x, x.x, fmaf(x.y, x.y, kk)); qq = fmaf(y.x, y.x, fmaf(y.y, y.y, qq));
      }
    }
    kk += __shfl_xor_sync(0xffffffffu, kk, 1); kk += __shfl_xor_sync(0xffffffffu, kk, 2);
    qq += __shfl_xor_sync(0xffffffffu, qq, 1); qq += __shfl_xor_sync(0xffffffffu, qq, 2);
    if (part == 0) { s_kn[r] = rsqrtf(kk + 1e-6f); s_qn[r] = rsqrtf(qq + 1e-6f) * rsqrtf((float)kDcD); }
  }
  // warps 0-3: K K^T, warps 4-7: Q K^T; 16 rows each, columns up to the diagonal
  const int j = warp & 3;
  float acc[8][4];
#pragma unroll
  for (int n = 0; n < 8; n++)
#pragma unroll
    for (int e = 0; e < 4; e++) acc[n][e] = 0.f;
#pragma unroll
  for (int kt = 0; kt < 8; kt++) {
    uint32_t fa[4];
    ldsm4(fa, dc_at(warp < 4 ? sK : sQ, j * 16 + (lane & 15), 2 * kt + (lane >> 4)));
#pragma unroll
    for (int i = 0; i < 4; i++) {
      if (i > j) continue;
      uint32_t fb[4];
      ldsm4(fb, dc_at(sK, i * 16 + (lane & 7) + ((lane >> 4) << 3), 2 * kt + ((lane >> 3) & 1)));
      mma_bf16(acc[2 * i], fa, fb[0], fb[1]);
      mma_bf16(acc[2 * i + 1], fa, fb[2], fb[3]);
    }
  }
  __syncthreads();            // norms are there; K and Q are no longer needed
#pragma unroll
  for (int n = 0; n < 8; n++) {
    if ((n >> 1) > j) continue;
#pragma unroll
    for (int e = 0; e < 4; e++) {
      const int t = j * 16 + (lane >> 2) + (e >> 1) * 8, c = n * 8 + (lane & 3) * 2 + (e & 1);
      const float f = acc[n][e] * s_kn[c] * expf((float)(s_g[t] - s_g[c]));
      if (warp < 4) sA[t * kDcLd + c] = c < t ? f * (s_b[t] * s_kn[t]) : 0.f;
      else sP[t * kDcLd + c] = c <= t ? f * s_qn[t] : 0.f;
    }
  }
  for (int i = tid; i < kDcC * kDcLd; i += kDcThreads) sT[i] = 0.f;
  __syncthreads();
  // T = (I + A)^-1: 16 x 16 on the diagonal by substitution, a column per thread
  if (tid < kDcC) {
    const int blk = tid >> 4, c = tid & 15;
    const float* A = sA + blk * 16 * (kDcLd + 1);
    float x[16];
#pragma unroll
    for (int i = 0; i < 16; i++) {
      float s = i == c ? 1.f : 0.f;
#pragma unroll
      for (int l = 0; l < i; l++) s = fmaf(-A[i * kDcLd + l], x[l], s);
      x[i] = s;
    }
#pragma unroll
    for (int i = 0; i < 16; i++) sT[(blk * 16 + i) * kDcLd + blk * 16 + c] = x[i];
  }
  __syncthreads();
  // [T11 0; -T22 A21 T11, T22] for 32 x 32, then for 64 x 64
  for (int i = tid; i < 512; i += kDcThreads) {
    const int p = i >> 8, r = (i >> 4) & 15, c = i & 15, o = p * 32;
    float s = 0.f;
#pragma unroll
    for (int l = 0; l < 16; l++) s = fmaf(sA[(o + 16 + r) * kDcLd + o + l], sT[(o + l) * kDcLd + o + c], s);
    sM[(p * 16 + r) * 33 + c] = s;
  }
  __syncthreads();
  for (int i = tid; i < 512; i += kDcThreads) {
    const int p = i >> 8, r = (i >> 4) & 15, c = i & 15, o = p * 32;
    float s = 0.f;
#pragma unroll
    for (int l = 0; l < 16; l++) s = fmaf(sT[(o + 16 + r) * kDcLd + o + 16 + l], sM[(p * 16 + l) * 33 + c], s);
    sT[(o + 16 + r) * kDcLd + o + c] = -s;
  }
  __syncthreads();
  for (int i = tid; i < 1024; i += kDcThreads) {
    const int r = i >> 5, c = i & 31;
    float s = 0.f;
#pragma unroll 8
    for (int l = 0; l < 32; l++) s = fmaf(sA[(32 + r) * kDcLd + l], sT[l * kDcLd + c], s);
    sM[r * 33 + c] = s;
  }
  __syncthreads();
  for (int i = tid; i < 1024; i += kDcThreads) {
    const int r = i >> 5, c = i & 31;
    float s = 0.f;
#pragma unroll 8
    for (int l = 0; l < 32; l++) s = fmaf(sT[(32 + r) * kDcLd + 32 + l], sM[l * 33 + c], s);
    sT[(32 + r) * kDcLd + c] = -s;
  }
  __syncthreads();
  // P T into A's place, 4 x 4 a thread
  {
    const int ty = tid >> 4, tx = tid & 15;
    float s[4][4] = {};
    if (tx <= ty)
      for (int l = tx * 4; l < ty * 4 + 4; l++) {
        const float4 t = *reinterpret_cast<const float4*>(sT + l * kDcLd + tx * 4);
#pragma unroll
        for (int r = 0; r < 4; r++) {
          const float p = sP[(ty * 4 + r) * kDcLd + l];
          s[r][0] = fmaf(p, t.x, s[r][0]); s[r][1] = fmaf(p, t.y, s[r][1]); s[r][2] = fmaf(p, t.z, s[r][2]); s[r][3] = fmaf(p, t.w, s[r][3]);
        }
      }
#pragma unroll
    for (int r = 0; r < 4; r++) *reinterpret_cast<float4*>(sA + (ty * 4 + r) * kDcLd + tx * 4) = make_float4(s[r][0], s[r][1], s[r][2], s[r][3]);
  }
  __syncthreads();
  const long long slot = (long long)blockIdx.x * a.Hv + h;
  uint8_t* frag = a.frags + slot * kDcFragBytes;
  for (int i = warp; i < 2 * kDcPairs; i += 8) {
    const bool pt = i >= kDcPairs;
    const int p = pt ? i - kDcPairs : i, jj = p < 1 ? 0 : p < 3 ? 1 : p < 6 ? 2 : 3, ii = p - jj * (jj + 1) / 2;
    const float* src = (pt ? sA : sT) + (jj * 16 + (lane >> 2)) * kDcLd + ii * 16 + (lane & 3) * 2;
    uint32_t w[3][4];
#pragma unroll
    for (int n = 0; n < 2; n++)
#pragma unroll
      for (int r = 0; r < 2; r++) {
        const float2 f = *reinterpret_cast<const float2*>(src + n * 8 * kDcLd + r * 8);
        split3(f.x, f.y, w[0][n * 2 + r], w[1][n * 2 + r], w[2][n * 2 + r]);
      }
    uint4* dst = reinterpret_cast<uint4*>(frag + i * 3 * 512) + lane;
#pragma unroll
    for (int t = 0; t < 3; t++) dst[32 * t] = make_uint4(w[t][0], w[t][1], w[t][2], w[t][3]);
  }
  if (tid < kDcC) {
    const float e = expf((float)s_g[tid]), b = s_b[tid];
    a.rows[slot * kDcC + tid] = make_float4(b, b * s_kn[tid] * e, s_qn[tid] * e, s_kn[tid] * expf((float)(s_g[kDcC - 1] - s_g[tid])));
    if (tid == 0) a.decay[slot] = expf((float)s_g[kDcC - 1]);
  }
}

constexpr int kDcN = 32;                       // value columns per CTA
constexpr int kDcM = kDcN / 16;
// shared memory of the scan: [2][K | Q] of 64 x 256 B | [2] V of 64 x 64 B | operand fragments of S (and, behind its last use, of U) | of R | [2] row factors
constexpr int kDcOffV = 4 * kDcC * 256, kDcOffS = kDcOffV + 2 * kDcC * kDcN * 2, kDcOffR = kDcOffS + 8 * kDcM * 3 * 512, kDcOffF = kDcOffR + 4 * kDcM * 3 * 512,
              kDcScanSmem = kDcOffF + 2 * kDcC * 16 + 128;

__global__ void __launch_bounds__(kDcThreads, 2) delta_chunk_scan_kernel(const DcArgs a) {
  pdl_wait(); pdl_trigger();
  extern __shared__ __align__(16) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~uintptr_t(127));
  const uint32_t base = smem_u32(smem), sS = base + kDcOffS, sR = base + kDcOffR, sF = base + kDcOffF;
  constexpr int kParts = kDcD / kDcN;
  const int seq = blockIdx.y, h = blockIdx.x / kParts, dv0 = (blockIdx.x % kParts) * kDcN, hk = h / (a.Hv / a.Hk);
  const int start = a.cu[seq], n = a.cu[seq + 1] - start;
  if (n < a.min_n || n <= 0) return;
  const int st_slot = a.slots[seq];
  if (!NE_INDEX_OK(st_slot, BK_STATE_SLOTS, kKernelDc, __LINE__)) return;
  // j: the warp's 16 tokens of a chunk; row block j of T or P T has j + 1 products, so a scheduler's two warps (w and w + 4) take j and 3 - j (600 -> 571 us)
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, j = warp < 4 ? warp : 7 - warp, g = lane >> 2, c2 = (lane & 3) * 2;
  int chunk0 = 0;             // chunks of the sequences in front
  for (int s0 = lane; s0 < seq; s0 += 32) chunk0 += (a.cu[s0 + 1] - a.cu[s0] + kDcC - 1) / kDcC;
  chunk0 = __reduce_add_sync(0xffffffffu, chunk0);

  // state: S^T as accumulators, rows = value columns, this warp's 16 key columns
  float* Sg = a.state + (((long long)st_slot * a.Hv + h) * kDcD + dv0) * kDcD;
  float S[kDcM][2][4];
  const bool have = a.fresh[seq] == 0;
#pragma unroll
  for (int m = 0; m < kDcM; m++)
#pragma unroll
    for (int x = 0; x < 2; x++)
#pragma unroll
      for (int r = 0; r < 2; r++) {
        const float2 f = have ? *reinterpret_cast<const float2*>(Sg + (m * 16 + g + r * 8) * kDcD + warp * 16 + x * 8 + c2) : make_float2(0.f, 0.f);
        S[m][x][2 * r] = f.x; S[m][x][2 * r + 1] = f.y;
      }
  // accumulators (rows x 16 columns) as the A operand of the next product, columns k-tile `kt`
  auto put = [&](uint32_t dst, int kt, const float (&d)[kDcM][2][4]) {
#pragma unroll
    for (int m = 0; m < kDcM; m++) {
      uint32_t w[3][4];
#pragma unroll
      for (int x = 0; x < 2; x++)
#pragma unroll
        for (int r = 0; r < 2; r++) split3(d[m][x][2 * r], d[m][x][2 * r + 1], w[0][2 * x + r], w[1][2 * x + r], w[2][2 * x + r]);
#pragma unroll
      for (int t = 0; t < 3; t++)
        *reinterpret_cast<uint4*>(smem + (dst - base) + ((kt * kDcM + m) * 3 + t) * 512 + lane * 16) = make_uint4(w[t][0], w[t][1], w[t][2], w[t][3]);
    }
  };
  auto get = [&](uint32_t src, int kt, int m, int t, uint32_t (&f)[4]) {
    const uint4 u = ld_shared_v4(src + ((kt * kDcM + m) * 3 + t) * 512 + lane * 16);
    f[0] = u.x; f[1] = u.y; f[2] = u.z; f[3] = u.w;
  };
  auto load = [&](int i0, int buf) {
    const int m = min(kDcC, n - i0);
    const long long t0 = start + i0;
    dc_load(base + buf * 2 * kDcC * 256, a.k + t0 * a.qk_ld + hk * kDcD, a.qk_ld, m);
    dc_load(base + (buf * 2 + 1) * kDcC * 256, a.q + t0 * a.qk_ld + hk * kDcD, a.qk_ld, m);
    {
      const int r = tid >> 2, p = tid & 3;
      cp_async16(base + kDcOffV + buf * kDcC * kDcN * 2 + r * kDcN * 2 + p * 16, a.v + (t0 + (r < m ? r : 0)) * a.v_ld + (long long)h * kDcD + dv0 + p * 8, r < m ? 16 : 0);
    }
    if (tid < kDcC) cp_async16(sF + buf * kDcC * 16 + tid * 16, a.rows + ((long long)(chunk0 + i0 / kDcC) * a.Hv + h) * kDcC + tid, 16);
    cp_async_commit();
  };
  load(0, 0);
  put(sS, warp, S);
  for (int i0 = 0, buf = 0; i0 < n; i0 += kDcC, buf ^= 1) {
    const long long slot = (long long)(chunk0 + i0 / kDcC) * a.Hv + h;
    const uint8_t* frag = a.frags + slot * kDcFragBytes;
    const float dec = a.decay[slot];
    cp_async_wait<0>();
    __syncthreads();          // the chunk's rows and the state's fragments are there, the other buffer is free
    if (i0 + kDcC < n) load(i0 + kDcC, buf ^ 1);
    const uint32_t sK = base + buf * 2 * kDcC * 256, sX = warp < 4 ? sK : sK + kDcC * 256;
    // this warp's 16 rows of T or P T
    uint4 fb[4][3];
#pragma unroll
    for (int kt = 0; kt < 4; kt++)
      if (kt <= j)
#pragma unroll
        for (int t = 0; t < 3; t++) fb[kt][t] = __ldg(reinterpret_cast<const uint4*>(frag + (((warp < 4 ? 0 : kDcPairs) + dc_pair(j, kt)) * 3 + t) * 512) + lane);
    // ---- S K^T and S Q^T: columns = this warp's 16 tokens
    float D[kDcM][2][4] = {};
#pragma unroll
    for (int kt = 0; kt < 8; kt++) {
      uint32_t b[4];
      ldsm4(b, dc_at(sX, j * 16 + (lane & 7) + ((lane >> 4) << 3), 2 * kt + ((lane >> 3) & 1)));
#pragma unroll
      for (int m = 0; m < kDcM; m++)
#pragma unroll
        for (int t = 0; t < 3; t++) {
          uint32_t f[4];
          get(sS, kt, m, t, f);
          mma_bf16(D[m][0], f, b[0], b[1]);
          mma_bf16(D[m][1], f, b[2], b[3]);
        }
    }
    const float4* rows = reinterpret_cast<const float4*>(smem + kDcOffF + buf * kDcC * 16) + j * 16;
    const __nv_bfloat16* sV = reinterpret_cast<const __nv_bfloat16*>(smem + kDcOffV + buf * kDcC * kDcN * 2) + j * 16 * kDcN;
    // ---- R = b (V - e^G K S^T) for the next product; outputs keep e^G Q S^T
#pragma unroll
    for (int x = 0; x < 2; x++)
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const int t = x * 8 + c2 + e;
        const float4 f = rows[t];
#pragma unroll
        for (int m = 0; m < kDcM; m++)
#pragma unroll
          for (int r = 0; r < 2; r++) {
            float& d = D[m][x][2 * r + e];
            d = warp < 4 ? f.x * __bfloat162float(sV[t * kDcN + m * 16 + g + r * 8]) - f.y * d : f.z * d;
          }
      }
    if (warp < 4) put(sR, j, D);
    __syncthreads();          // R is there; nobody reads the state's fragments any more
    // ---- U = T R (outputs: P T R)
    float U[kDcM][2][4] = {};
#pragma unroll
    for (int kt = 0; kt < 4; kt++) {
      if (kt > j) continue;
#pragma unroll
      for (int m = 0; m < kDcM; m++) {
        uint32_t f[3][4];
#pragma unroll
        for (int t = 0; t < 3; t++) get(sR, kt, m, t, f[t]);
        // smallest products first
#pragma unroll
        for (int s = 2; s >= 0; s--)
#pragma unroll
          for (int t = 0; t <= s; t++) {
            mma_bf16(U[m][0], f[t], fb[kt][s - t].x, fb[kt][s - t].y);
            mma_bf16(U[m][1], f[t], fb[kt][s - t].z, fb[kt][s - t].w);
          }
      }
    }
    if (warp < 4) {
#pragma unroll
      for (int x = 0; x < 2; x++)
#pragma unroll
        for (int e = 0; e < 2; e++) {
          const float w = rows[x * 8 + c2 + e].w;
#pragma unroll
          for (int m = 0; m < kDcM; m++) { U[m][x][e] *= w; U[m][x][2 + e] *= w; }
        }
      put(sS, j, U);
    } else {
#pragma unroll
      for (int m = 0; m < kDcM; m++)
#pragma unroll
        for (int x = 0; x < 2; x++)
#pragma unroll
          for (int e = 0; e < 4; e++) D[m][x][e] += U[m][x][e];
    }
    __syncthreads();          // U is there
    // ---- S = e^(G_C) S + (e^(G_C - G) U)^T K
    float W[kDcM][2][4] = {};
#pragma unroll
    for (int t = 2; t >= 0; t--)
#pragma unroll
      for (int kt = 0; kt < 4; kt++) {
        uint32_t b[4];
        ldsm4t(b, dc_at(sK, kt * 16 + (lane & 7) + ((lane >> 3) & 1) * 8, 2 * warp + (lane >> 4)));
#pragma unroll
        for (int m = 0; m < kDcM; m++) {
          uint32_t f[4];
          get(sS, kt, m, t, f);
          mma_bf16(W[m][0], f, b[0], b[1]);
          mma_bf16(W[m][1], f, b[2], b[3]);
        }
      }
#pragma unroll
    for (int m = 0; m < kDcM; m++)
#pragma unroll
      for (int x = 0; x < 2; x++)
#pragma unroll
        for (int e = 0; e < 4; e++) S[m][x][e] = fmaf(S[m][x][e], dec, W[m][x][e]);
    if (warp >= 4) {
      const int left = n - i0 - j * 16;
      float* o = a.raw + ((long long)(start + i0 + j * 16) * a.Hv + h) * kDcD + dv0 + g;
#pragma unroll
      for (int x = 0; x < 2; x++)
#pragma unroll
        for (int e = 0; e < 2; e++) {
          const int t = x * 8 + c2 + e;
          if (t < left)
#pragma unroll
            for (int m = 0; m < kDcM; m++) {
              o[(long long)t * a.Hv * kDcD + m * 16] = D[m][x][e];
              o[(long long)t * a.Hv * kDcD + m * 16 + 8] = D[m][x][2 + e];
            }
        }
    }
    __syncthreads();          // U's fragments have been read
    put(sS, warp, S);
  }
#pragma unroll
  for (int m = 0; m < kDcM; m++)
#pragma unroll
    for (int x = 0; x < 2; x++)
#pragma unroll
      for (int r = 0; r < 2; r++)
        *reinterpret_cast<float2*>(Sg + (m * 16 + g + r * 8) * kDcD + warp * 16 + x * 8 + c2) = make_float2(S[m][x][2 * r], S[m][x][2 * r + 1]);
}

constexpr int kDcPrepSmem = 2 * kDcC * 256 + 2 * kDcC * kDcLd * 4 + 128;
static_assert((kDcC * kDcLd + 32 * 33) * 4 <= 2 * kDcC * 256, "T and the intermediate fit over K and Q");

}  // namespace ne

using namespace ne;

// Bytes of workspace per chunk and head: fragments, row factors, decay.  Chunks: at most T / 64 + B.
extern "C" long long ne_delta_chunk_work(void) { return kDcFragBytes + kDcC * 16 + 16; }

// Sequences of at least min_n tokens in this call (the others are left alone): arguments as ne_gdn_step's, 128 x 128 states, rows of q, k, v on 16-byte
// boundaries.  work: chunks x Hv x ne_delta_chunk_work() bytes; raw fp32 [T, Hv, 128].
extern "C" int ne_delta_chunk(const void* q, const void* k, const void* v, long long qk_ld, long long v_ld, const void* a, const void* b, long long ab_ld,
                              const float* A_log, const float* dt_bias, float* state, const int* slots, const int* cu, const int* fresh, float* raw, void* work,
                              int T, int B, int chunks, int Hk, int Hv, int min_n, cudaStream_t st) {
  if (T <= 0 || B <= 0) return 0;
  if (Hk < 1 || Hv % Hk || Hv > 65535 || B > 65535 || chunks < 1) return 1001;
  if (qk_ld % 8 || v_ld % 8 || (((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)work) & 15)) return 1002;
  DcArgs x;
  x.q = (const __nv_bfloat16*)q; x.k = (const __nv_bfloat16*)k; x.v = (const __nv_bfloat16*)v; x.qk_ld = qk_ld; x.v_ld = v_ld;
  x.a = (const __nv_bfloat16*)a; x.b = (const __nv_bfloat16*)b; x.ab_ld = ab_ld; x.A_log = A_log; x.dt_bias = dt_bias; x.state = state; x.slots = slots; x.cu = cu;
  x.fresh = fresh; x.raw = raw; x.num_seqs = B; x.Hk = Hk; x.Hv = Hv; x.min_n = min_n;
  const long long cells = (long long)chunks * Hv;
  x.frags = (uint8_t*)work; x.rows = (float4*)(x.frags + cells * kDcFragBytes); x.decay = (float*)(x.rows + cells * kDcC);
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(delta_chunk_prepare_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kDcPrepSmem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(delta_chunk_scan_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kDcScanSmem);
    if (e != cudaSuccess) return (int)e;
    configured = true;
  }
  cudaError_t e = launch_pdl(delta_chunk_prepare_kernel, dim3((unsigned)chunks, (unsigned)Hv), dim3(kDcThreads), kDcPrepSmem, st, x);
  if (e != cudaSuccess) return (int)e;
  return (int)launch_pdl(delta_chunk_scan_kernel, dim3((unsigned)(Hv * (kDcD / kDcN)), (unsigned)B), dim3(kDcThreads), kDcScanSmem, st, x);
}
