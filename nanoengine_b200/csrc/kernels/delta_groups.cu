// The gated delta rule over portions of a few tokens and more, four tokens at a time, 128 x 128 states, everything in 32-bit: a log-decay per key channel
// (Kimi delta attention, any length) or per head (gated delta net, portions too short for delta_chunk.cu).
//     S <- S diag(e^g),  u = b (v - S k),  S <- S + u k^T,  o = S q      (k, q unit vectors, q scaled by 128^-0.5)
// Rows of a state are independent of each other, so a CTA takes 64 of the 128 rows of one (sequence, head), in registers: eight lanes share a row, 16 columns
// each, a warp holds 16 rows.  With d_t = e^(g_t), E_ts = d_(s+1) .. d_t (products of factors of at most one: nothing to cancel or overflow) a group's
//     w_t = S (E_t0 d_0 k_t),  u_t = b_t (v_t - w_t - sum_(s<t) A_ts u_s),   A_ts = k_t . E_ts k_s
//     o_t = S (E_t0 d_0 q_t) + sum_(s<=t) P_ts u_s,                          P_ts = q_t . E_ts k_s
//     S <- S diag(E_30 d_0) + sum_s u_s (E_3s k_s)^T
// take 13 operations per state element where token by token takes 16, and one reduction over the eight lanes in a row where it takes four.  The vectors and
// the 16 scalars of a group are made by one warp, sixteen tokens (four groups) at a time, in shared memory; their rows arrive by asynchronous copies while the
// sixteen before are worked on.  A reduction leaves every lane with its share of the sums (14 exchanges for 16 sums, not 48).
// FMA pipe and shared memory are needed about equally (832 cycles a group and head half on an SM each).  Measured: per channel, 6 prompts of 500 .. 1500
// tokens, 32 heads: 2690 -> 926 us (before: gdn.cu's kernel, token by token, 40 exchanges of a whole warp a token); error of the final state against 64 bits
// 2.2e-7 (before: 8.8e-7).  Per head from 64 tokens on delta_chunk.cu has the smaller error and, from 300, the shorter time.
//
// Replaces in the reference: layers/backends/delta_net/kda.py:300-377.
#include "ptx.cuh"

namespace ne {

[[maybe_unused]] constexpr int kKernelDg = 29;      // in status words of the checked build
constexpr int kDgTok = 16;                     // tokens per stage
constexpr int kDgRows = 64;                    // state rows per CTA
constexpr int kDgThreads = 128;
typedef unsigned long long f32x2;

struct DgArgs {
  const __nv_bfloat16* q; const __nv_bfloat16* k; const __nv_bfloat16* v; const __nv_bfloat16* g; const __nv_bfloat16* b;
  long long qk_ld, v_ld, g_ld, b_ld;           // g: [T, H, 128] contiguous (per channel) or rows of at least H
  const float* A_log; const float* dt_bias; float lower_bound;
  float* state; const int* slots; const int* cu; const int* fresh; float* raw;
  int B, H, rep, min_n, max_n;
};

__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) { f32x2 d; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c)); return d; }
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) { f32x2 d; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
__device__ __forceinline__ f32x2 both(float x) { f32x2 d; asm("mov.b64 %0, {%1, %1};" : "=l"(d) : "f"(x)); return d; }
__device__ __forceinline__ float sum2(f32x2 a) { float x, y; asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a)); return x + y; }
__device__ __forceinline__ float pick(const float (&x)[4], int i) { return i & 2 ? (i & 1 ? x[3] : x[2]) : (i & 1 ? x[1] : x[0]); }

constexpr int kDgVecs = 13;                    // of a group: 4 decayed k, 4 decayed q, 4 k decayed to the group's end, the whole decay
// shared memory: [2] raw rows k | q | g (256 B a token) | v (128 B a token); then the vectors of four groups, fp32
constexpr int kDgRaw = kDgTok * (3 * 256 + kDgRows * 2), kDgSmem = 2 * kDgRaw + 4 * kDgVecs * 512;

// 16 sums [token][row] over the eight lanes of a row: lane sub ends with row sub & 3, tokens 2 (sub >> 2) and the next
__device__ __forceinline__ void reduce16(const float (&x)[4][4], int sub, float (&w)[2]) {
  float y[2][4], z[2][2];
#pragma unroll
  for (int t = 0; t < 2; t++)
#pragma unroll
    for (int r = 0; r < 4; r++) y[t][r] = (sub & 4 ? x[2 + t][r] : x[t][r]) + __shfl_xor_sync(0xffffffffu, sub & 4 ? x[t][r] : x[2 + t][r], 4);
#pragma unroll
  for (int t = 0; t < 2; t++)
#pragma unroll
    for (int r = 0; r < 2; r++) z[t][r] = (sub & 2 ? y[t][2 + r] : y[t][r]) + __shfl_xor_sync(0xffffffffu, sub & 2 ? y[t][r] : y[t][2 + r], 2);
#pragma unroll
  for (int t = 0; t < 2; t++) w[t] = (sub & 1 ? z[t][1] : z[t][0]) + __shfl_xor_sync(0xffffffffu, sub & 1 ? z[t][0] : z[t][1], 1);
}

// blockIdx.x's half head of a sequence
template <bool kVec>
__device__ __forceinline__ void delta_groups_sequence(const DgArgs& a, int seq, uint8_t* smem_raw) {
  __shared__ float s_beta[kDgTok], s_A[4][8];
  __shared__ float4 s_P[4][4];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, grp = lane >> 3, sub = lane & 7;
  const int h = blockIdx.x >> 1, row0 = (blockIdx.x & 1) * kDgRows, hk = h / a.rep;
  const int start = a.cu[seq], n = a.cu[seq + 1] - start;
  const int slot = a.slots[seq];
  if (!NE_INDEX_OK(slot, BK_STATE_SLOTS, kKernelDg, __LINE__)) return;
  // lane: rows row0 + warp 16 + r 4 + grp, columns i 32 + sub 4 ..
  float* Sg = a.state + (((long long)slot * a.H + h) * 128 + row0 + warp * 16 + grp) * 128 + sub * 4;
  f32x2 S[4][8];
  const bool have = a.fresh[seq] == 0;
#pragma unroll
  for (int r = 0; r < 4; r++)
#pragma unroll
    for (int i = 0; i < 4; i++) {
      ulonglong2 x = make_ulonglong2(0ull, 0ull);
      if (have) x = *reinterpret_cast<const ulonglong2*>(Sg + r * 4 * 128 + i * 32);
      S[r][2 * i] = x.x; S[r][2 * i + 1] = x.y;
    }
  const float expA = expf(a.A_log[h]);
  float bias[kVec ? 4 : 1];
#pragma unroll
  for (int e = 0; e < (kVec ? 4 : 1); e++) bias[e] = a.dt_bias[kVec ? h * 128 + lane * 4 + e : h];
  auto log_decay = [&](float x) {
    return kVec && a.lower_bound < 0.f ? a.lower_bound / (1.f + expf(-expA * x)) : -expA * (x > 20.f ? x : log1pf(expf(x)));
  };
  float* conv = reinterpret_cast<float*>(smem_raw + 2 * kDgRaw);       // [group][kDgVecs][128]
  const uint32_t base = smem_u32(smem_raw);
  auto load = [&](int i0, int buf) {           // rows past the end are zero
    const int m = min(kDgTok, n - i0);
    const uint32_t dst = base + buf * kDgRaw;
#pragma unroll
    for (int i = tid; i < kDgTok * 16; i += kDgThreads) {
      const int t = i >> 4, p = i & 15, bytes = t < m ? 16 : 0;
      const long long row = start + i0 + (t < m ? t : 0);
      cp_async16(dst + t * 256 + p * 16, a.k + row * a.qk_ld + hk * 128 + p * 8, bytes);
      cp_async16(dst + (kDgTok + t) * 256 + p * 16, a.q + row * a.qk_ld + hk * 128 + p * 8, bytes);
      if (kVec) cp_async16(dst + (2 * kDgTok + t) * 256 + p * 16, a.g + (row * a.H + h) * 128 + p * 8, bytes);
    }
    {
      const int t = tid >> 3, p = tid & 7;
      cp_async16(dst + 3 * kDgTok * 256 + t * 128 + p * 16, a.v + (start + i0 + (t < m ? t : 0)) * a.v_ld + h * 128 + row0 + p * 8, t < m ? 16 : 0);
    }
    cp_async_commit();
  };
  // gates of this warp's group: lane t < 4 holds token t's
  float b_raw = 0.f, g_raw = 0.f;
  auto gates = [&](int i0) {
    const int t = i0 + warp * 4 + lane;
    if (lane < 4 && t < n) {
      b_raw = __bfloat162float(a.b[(long long)(start + t) * a.b_ld + h]);
      if (!kVec) g_raw = __bfloat162float(a.g[(long long)(start + t) * a.g_ld + h]);
    }
  };
  load(0, 0);
  gates(0);
  for (int i0 = 0, buf = 0; i0 < n; i0 += kDgTok, buf ^= 1) {
    const int m = min(kDgTok, n - i0);
    cp_async_wait<0>();
    __syncthreads();          // this stage's rows are there; the stage before has been worked on
    const uint8_t* raw = smem_raw + buf * kDgRaw;
    const int mine = i0 + warp * 4;            // this warp's group
    const float beta_l = mine + lane < n ? 1.f / (1.f + expf(-b_raw)) : 0.f;
    const float d_l = !kVec && mine + lane < n ? expf(log_decay(g_raw + bias[0])) : 1.f;
    if (i0 + kDgTok < n) { load(i0 + kDgTok, buf ^ 1); gates(i0 + kDgTok); }
    if (lane < 4) s_beta[warp * 4 + lane] = beta_l;
    if (warp * 4 < m) {
      float k[4][4], q[4][4], d[4][4];
#pragma unroll
      for (int t = 0; t < 4; t++) {
        const int o = (warp * 4 + t) * 256 + lane * 8;
        const uint2 uk = *reinterpret_cast<const uint2*>(raw + o), uq = *reinterpret_cast<const uint2*>(raw + kDgTok * 256 + o);
        const float2 k0 = unpack_bf16x2(uk.x), k1 = unpack_bf16x2(uk.y), q0 = unpack_bf16x2(uq.x), q1 = unpack_bf16x2(uq.y);
        k[t][0] = k0.x; k[t][1] = k0.y; k[t][2] = k1.x; k[t][3] = k1.y;
        q[t][0] = q0.x; q[t][1] = q0.y; q[t][2] = q1.x; q[t][3] = q1.y;
        if constexpr (kVec) {
          const uint2 ug = *reinterpret_cast<const uint2*>(raw + 2 * kDgTok * 256 + o);
          const float2 g0 = unpack_bf16x2(ug.x), g1 = unpack_bf16x2(ug.y);
          const float x[4] = {g0.x, g0.y, g1.x, g1.y};
#pragma unroll
          for (int e = 0; e < 4; e++) d[t][e] = mine + t < n ? expf(log_decay(x[e] + bias[e])) : 1.f;
        } else {
          const float x = __shfl_sync(0xffffffffu, d_l, t);
#pragma unroll
          for (int e = 0; e < 4; e++) d[t][e] = x;
        }
      }
      // 0-3: k.k, 4-7: q.q, 8-13: A (t, s < t), 14-23: P (t, s <= t), from the rows as they are
      float x[32];
#pragma unroll
      for (int i = 0; i < 32; i++) x[i] = 0.f;
#pragma unroll
      for (int e = 0; e < 4; e++) {
#pragma unroll
        for (int t = 0; t < 4; t++) {
          x[t] = fmaf(k[t][e], k[t][e], x[t]);
          x[4 + t] = fmaf(q[t][e], q[t][e], x[4 + t]);
          float f = 1.f;
#pragma unroll
          for (int s = t; s >= 0; s--) {       // f = d_(s+1) .. d_t
            if (s < t) { f *= d[s + 1][e]; x[8 + t * (t - 1) / 2 + s] = fmaf(k[t][e] * f, k[s][e], x[8 + t * (t - 1) / 2 + s]); }
            x[14 + t * (t + 1) / 2 + s] = fmaf(q[t][e] * f, k[s][e], x[14 + t * (t + 1) / 2 + s]);
          }
        }
      }
      // lane i ends with sum i
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int i = 0; i < o; i++) x[i] = (lane & o ? x[o + i] : x[i]) + __shfl_xor_sync(0xffffffffu, lane & o ? x[i] : x[o + i], o);
      const float norm = rsqrtf(x[0] + 1e-6f) * (lane & 4 ? rsqrtf(128.f) : 1.f);
      float kn[4], qn[4];
#pragma unroll
      for (int t = 0; t < 4; t++) { kn[t] = __shfl_sync(0xffffffffu, norm, t); qn[t] = __shfl_sync(0xffffffffu, norm, 4 + t); }
      if (lane >= 8 && lane < 24) {
        // (t, s) of lanes 8..23, two bits each: A 10 20 21 30 31 32, P 00 10 11 20 21 22 30 31 32 33
        const int i = (lane - 8) * 2, t = (0xffa94fe9u >> i) & 3, s = (0xe4910910u >> i) & 3;
        const float c = x[0] * (lane < 14 ? pick(kn, t) : pick(qn, t)) * pick(kn, s);
        if (lane < 14) s_A[warp][lane - 8] = c;
        else reinterpret_cast<float*>(&s_P[warp][t])[s] = c;
      }
      float* dst = conv + warp * kDgVecs * 128 + lane * 4;
      float f[4] = {1.f, 1.f, 1.f, 1.f};
#pragma unroll
      for (int t = 0; t < 4; t++) {
#pragma unroll
        for (int e = 0; e < 4; e++) f[e] *= d[t][e];
        *reinterpret_cast<float4*>(dst + t * 128) = make_float4(f[0] * k[t][0] * kn[t], f[1] * k[t][1] * kn[t], f[2] * k[t][2] * kn[t], f[3] * k[t][3] * kn[t]);
        *reinterpret_cast<float4*>(dst + (4 + t) * 128) = make_float4(f[0] * q[t][0] * qn[t], f[1] * q[t][1] * qn[t], f[2] * q[t][2] * qn[t], f[3] * q[t][3] * qn[t]);
      }
      *reinterpret_cast<float4*>(dst + 12 * 128) = make_float4(f[0], f[1], f[2], f[3]);
#pragma unroll
      for (int e = 0; e < 4; e++) f[e] = 1.f;
#pragma unroll
      for (int t = 3; t >= 0; t--) {
        *reinterpret_cast<float4*>(dst + (8 + t) * 128) = make_float4(f[0] * k[t][0] * kn[t], f[1] * k[t][1] * kn[t], f[2] * k[t][2] * kn[t], f[3] * k[t][3] * kn[t]);
#pragma unroll
        for (int e = 0; e < 4; e++) f[e] *= d[t][e];
      }
    }
    __syncthreads();
    const __nv_bfloat16* sv = reinterpret_cast<const __nv_bfloat16*>(raw + 3 * kDgTok * 256) + warp * 16 + (sub & 3) * 4 + grp;
    float* out = a.raw + ((long long)(start + i0) * a.H + h) * 128 + row0 + warp * 16 + (sub & 3) * 4 + grp;
    for (int gi = 0; gi * 4 < m; gi++) {
      const ulonglong2* c = reinterpret_cast<const ulonglong2*>(conv + gi * kDgVecs * 128 + sub * 4);      // vector j, columns i 32 + sub 4: piece j 32 + i 8
      f32x2 acc[4][4];
      float x[4][4], w[2];
      auto dots = [&](int j0) {
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
          for (int t = 0; t < 4; t++) {
            const ulonglong2 y = c[(j0 + t) * 32 + i * 8];
#pragma unroll
            for (int r = 0; r < 4; r++) {
              acc[t][r] = i == 0 ? mul2(S[r][0], y.x) : fma2(S[r][2 * i], y.x, acc[t][r]);
              acc[t][r] = fma2(S[r][2 * i + 1], y.y, acc[t][r]);
            }
          }
#pragma unroll
        for (int t = 0; t < 4; t++)
#pragma unroll
          for (int r = 0; r < 4; r++) x[t][r] = sum2(acc[t][r]);
      };
      dots(0);
      reduce16(x, sub, w);
      float W[4];
      {
        const float o0 = __shfl_xor_sync(0xffffffffu, w[0], 4), o1 = __shfl_xor_sync(0xffffffffu, w[1], 4);
        W[0] = sub & 4 ? o0 : w[0]; W[1] = sub & 4 ? o1 : w[1]; W[2] = sub & 4 ? w[0] : o0; W[3] = sub & 4 ? w[1] : o1;
      }
      dots(4);
      float u[4];             // of row sub & 3
#pragma unroll
      for (int t = 0; t < 4; t++) {
        float y = __bfloat162float(sv[(gi * 4 + t) * kDgRows]) - W[t];
#pragma unroll
        for (int s = 0; s < t; s++) y = fmaf(-s_A[gi][t * (t - 1) / 2 + s], u[s], y);
        u[t] = y * s_beta[gi * 4 + t];
      }
      if (gi * 4 + 4 > m) {
#pragma unroll
        for (int t = 1; t < 4; t++)
          if (gi * 4 + t >= m) u[t] = 0.f;     // behind the end: nothing, whatever the state holds
      }
      reduce16(x, sub, w);
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const ulonglong2 D = c[12 * 32 + i * 8];
#pragma unroll
        for (int r = 0; r < 4; r++) { S[r][2 * i] = mul2(S[r][2 * i], D.x); S[r][2 * i + 1] = mul2(S[r][2 * i + 1], D.y); }
      }
#pragma unroll
      for (int t = 0; t < 4; t++) {
        f32x2 U[4];
#pragma unroll
        for (int r = 0; r < 4; r++) U[r] = both(__shfl_sync(0xffffffffu, u[t], (lane & 24) + r));
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const ulonglong2 y = c[(8 + t) * 32 + i * 8];
#pragma unroll
          for (int r = 0; r < 4; r++) { S[r][2 * i] = fma2(U[r], y.x, S[r][2 * i]); S[r][2 * i + 1] = fma2(U[r], y.y, S[r][2 * i + 1]); }
        }
      }
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const int t = (sub >> 2) * 2 + e;
        const float4 p = s_P[gi][t];
        float o = fmaf(p.x, u[0], w[e]);
        if (e == 1) o = fmaf(p.y, u[1], o);
        if (sub & 4) {                         // later tokens by a choice, not by a factor of zero: their u may be no number
          if (e == 0) o = fmaf(p.y, u[1], o);
          o = fmaf(p.z, u[2], o);
          if (e == 1) o = fmaf(p.w, u[3], o);
        }
        if (gi * 4 + t < m) out[(long long)(gi * 4 + t) * a.H * 128] = o;
      }
    }
  }
#pragma unroll
  for (int r = 0; r < 4; r++)
#pragma unroll
    for (int i = 0; i < 4; i++) *reinterpret_cast<ulonglong2*>(Sg + r * 4 * 128 + i * 32) = make_ulonglong2(S[r][2 * i], S[r][2 * i + 1]);
}

template <bool kVec>
__global__ void __launch_bounds__(kDgThreads, 3) delta_groups_kernel(const DgArgs a) {
  pdl_wait(); pdl_trigger();
  extern __shared__ __align__(16) uint8_t smem_raw[];
  const int lane = threadIdx.x & 31;
  // Of the sequences that are long enough the blockIdx.y-th, and every gridDim.y-th behind it.  Up to 64 in the order of their lengths, longest first: lanes hold a
  // number that grows with the length and tells equal ones apart, for two sequences each.  More as they come (so many fill the SMs several times over, and the
  // last wave weighs less), without counting where there is a CTA for each.
  auto length = [&](int s) { return s < a.B ? a.cu[s + 1] - a.cu[s] : 0; };
  auto fit = [&](int n) { return n >= a.min_n && n < a.max_n; };
  unsigned key[2] = {0, 0};
  if (a.B <= 64)
#pragma unroll
    for (int i = 0; i < 2; i++) { const int s = lane + 32 * i, n = length(s); if (fit(n)) key[i] = (unsigned)min(n, 1 << 25) << 6 | (63 - s); }
  int at = 0, from = 0, before = 0;            // as they come: sequences in front of `from` hold `before` that fit
  for (int y = blockIdx.y; y < a.B; y += gridDim.y) {
    int seq = -1;
    if (a.B <= 64) {
      unsigned top = 0;
      for (; at <= y; at++) {
        top = __reduce_max_sync(0xffffffffu, max(key[0], key[1]));
        if (!top) return;
        if (key[0] == top) key[0] = 0;
        if (key[1] == top) key[1] = 0;
      }
      seq = 63 - (int)(top & 63);
    } else if ((int)gridDim.y == a.B) {
      if (fit(length(y))) seq = y;
    } else {
      for (; from < a.B; from += 32) {
        const unsigned all = __ballot_sync(0xffffffffu, fit(length(from + lane)));
        if (y < before + __popc(all)) {
          seq = from + __ffs(__ballot_sync(0xffffffffu, (all >> lane & 1) && before + __popc(all & ((1u << lane) - 1)) == y)) - 1;
          break;
        }
        before += __popc(all);
      }
    }
    if (seq < 0) return;
    if (y != (int)blockIdx.y) __syncthreads();          // shared memory is the next one's
    delta_groups_sequence<kVec>(a, seq, smem_raw);
  }
}

}  // namespace ne

using namespace ne;

static int dg_sms() {
  static int n = 0;
  if (!n) { int dev; cudaGetDevice(&dev); cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev); }
  return n;
}

extern "C" int ne_gdn_step(const void* q, const void* k, const void* v, long long qk_ld, long long v_ld, const void* a, const void* b, long long ab_ld,
                           const float* A_log, const float* dt_bias, float* state, const int* slots, const int* cu, const int* fresh, const void* z,
                           long long z_ld, const void* norm_w, float eps, void* out, long long out_ld, int B, int Hk, int Hv, int Dk, int Dv, int skip_len,
                           int raw_out, int vec_gate, float lower_bound, cudaStream_t st);

// Sequences of less than max_n tokens in this call (the others are left alone): those of at least min_n (> 0) four tokens at a time, if `groups`, those of less
// token by token, if `step`, so that which form a sequence takes is its own length's matter and not its neighbours'.  q, k [T, Hk, 128] (row stride qk_ld),
// v [T, H, 128] (v_ld), b [T, >= H] (b_ld); per_channel: g [T, H, 128] contiguous, dt_bias [H, 128], log decays lower_bound sigmoid(e^A (g + bias)) if
// lower_bound < 0, else -e^A softplus(g + bias); otherwise g [T, >= H] (rows as b's), dt_bias [H], -e^A softplus.  Rows of q, k, v, per-channel g and the state on
// 16-byte boundaries.  raw fp32 [T, H, 128].
extern "C" int ne_delta_portions(const void* q, const void* k, const void* v, const void* g, const void* b, long long qk_ld, long long v_ld, long long b_ld,
                                 const float* A_log, const float* dt_bias, float lower_bound, float* state, const int* slots, const int* cu, const int* fresh,
                                 float* raw, int T, int B, int Hk, int H, int min_n, int max_n, int step, int groups, int per_channel, cudaStream_t st) {
  if (B <= 0) return 0;
  if (Hk < 1 || H % Hk || B > 65535 || min_n < 1) return 1001;
  if (qk_ld % 8 || v_ld % 8 || (((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)state) & 15) || (per_channel && ((uintptr_t)g & 15))) return 1002;
  if (step) {
    const int rc = ne_gdn_step(q, k, v, qk_ld, v_ld, g, b, b_ld, A_log, dt_bias, state, slots, cu, fresh, nullptr, 0, nullptr, 0.f, raw, (long long)H * 128, B, Hk, H,
                               128, 128, min(min_n, max_n), 1, per_channel, lower_bound, st);
    if (rc) return rc;
  }
  // No more than T / min_n can be long enough.  Where most sequences are shorter, a wave of CTAs, which then take several, costs less than one for each that may
  // find nothing to do: 64 portions of 2 tokens, 32 heads: 70 us against 77, without this kernel 68.
  const int rows = T >= min_n * B ? B : min(T / min_n, (3 * dg_sms() + 2 * H - 1) / (2 * H));
  if (!groups || rows < 1) return 0;
  DgArgs a;
  a.q = (const __nv_bfloat16*)q; a.k = (const __nv_bfloat16*)k; a.v = (const __nv_bfloat16*)v; a.g = (const __nv_bfloat16*)g; a.b = (const __nv_bfloat16*)b;
  a.qk_ld = qk_ld; a.v_ld = v_ld; a.g_ld = b_ld; a.b_ld = b_ld; a.A_log = A_log; a.dt_bias = dt_bias; a.lower_bound = lower_bound; a.state = state;
  a.slots = slots; a.cu = cu; a.fresh = fresh; a.raw = raw; a.B = B; a.H = H; a.rep = H / Hk; a.min_n = min_n; a.max_n = max_n;
  auto kern = per_channel ? delta_groups_kernel<true> : delta_groups_kernel<false>;
  static bool configured[2] = {false, false};
  if (!configured[per_channel != 0]) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kDgSmem);
    if (e != cudaSuccess) return (int)e;
    configured[per_channel != 0] = true;
  }
  return (int)launch_pdl(kern, dim3((unsigned)(2 * H), (unsigned)rows), dim3(kDgThreads), kDgSmem, st, a);
}
