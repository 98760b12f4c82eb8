// Prompt attention on tcgen05 tensor cores with the probabilities kept in TMEM: bf16 queries, keys and values, head sizes up to 256 in
// multiples of 8 (queries / keys and values may differ), any group of query heads per key / value head up to 128, causal or not, a window of the
// last keys; keys and values in 64-token cache pages, or as rows of the same ragged tokens (vision encoders, prompts without a cached prefix).
//
// One CTA = one KV head x up to two tiles of 128 (token, head of the group) rows of ONE sequence x one slice of its keys, in blocks of 64 keys (a page).
// Every tile t has two TMEM score slots of 64 columns (three where one tile has all of TMEM), block j in slot j mod their number, and a thread that issues its
// products in the order S(0) S(1), then PV(j) S(j+2) ..:
//     S(j) = Q K^T        (tcgen05.mma kind::f16, M = 128, N = 64, K = 16 steps up to the head size, so a head of 72 pays for 80)
//     P(j) = exp2(S - m)  one warpgroup per tile; bf16 pairs written over S(j) in TMEM, the A operand of the second product
//     O   += P(j) V       (N = head size up to the next multiple of 16; V read MN-major)
// The softmax finds S(j+1) ready when it has handed P(j) on.  (Blocks of 128 keys with one slot a tile read less shared memory per product, but then scores,
// softmax and products of a tile are one chain, whether one or two warpgroups share a tile's softmax: slower.  One tile per CTA and two CTAs per SM, or an issuer
// each for scores and products, were slower for long prompts too.)
// The order of two products is promised only where they share accumulator and shape, so S(j+2) waits for the products that read the slot: PV(j) itself with two
// slots, which the other tile's products, or the other CTA's, fill (1063 -> 1088 us for the MLA prompts below, against issuing without the wait), PV(j-1) with
// three (256-wide heads, nothing beside them: 177 without a wait, 197 with two slots, 186 so).
// A barrier test costs an issuing thread 300 cycles once products are queued before it, hence an issuer per tile, and tests in threes.
// kSplitP: a probability as a bf16 head and a bf16 remainder, both rounded, so it is off by 2^-17 of itself at most, to either side, and its sum takes it whole; two
// products against V.  Taken where the plain kernel this one replaced kept them in fp32: sums before they are rounded to bf16 are 2.7e-6 off (2-norm, 40 .. 3000
// keys; that kernel: 1e-7 .. 8e-7, a head that is cut off: 5e-6), the results 1.66e-3, as that kernel's.
// Shared memory: Q, then a ring of 8 KB slots (64 keys x 64 columns) shared by K and V, loaded in the order of first use; the chunks of a block's K
// or V (a group) share one barrier.
// Rows of V in front of the window or past the last visible key (pages that belong to nobody, rows of the next sequence: often no numbers) are zeroed in shared
// memory before their product: 0 x inf there would reach the result.  Values that some rows of a tile see and others do not: fmha_row_again.  Warp 0: TMA producer, 1 and 2: MMA issuers of tile 0 and 1, 3: that zeroing,
// 4-7 / 8-11: softmax, rescale and epilogue of tile 0 / 1.  All waits are bounded.
//
// Bound: the hand-overs between scores, softmax and products; no unit is full (busy % of the tensor pipe / exponentials / issue slots: MLA prompts 42 / 34 / 39,
// GQA 37 / 38 / 39, windows of 256-wide heads 43 / 15 / 24, vision 34 / 38 / 45).  Measured (B200, us, before -> so): 64 / 4 heads of 128, prompts of 1024 .. 3072
// tokens, 8192 in all: 574 -> 415 (gqa_bf16.cu, one tile, one CTA per SM); MLA, 128 heads, the same prompts: 1323 -> 1080 (that kernel); 16 / 4 heads of 256,
// window 1024, 6000 tokens: 51740 -> 157 and 16 heads of 72, 5 images of 600 .. 1800 patches: 143260 -> 116 (attn_generic.cu, a token and four heads per CTA on the
// CUDA cores).
//
// Replaces in the reference: the FA4 / FA3 varlen prefill calls (layers/backends/attention/fa4.py:34-245, fa3.py), the ragged MLA prefill of
// models/deepseek_v2/deepseek_v2.py:1792-1816, and the varlen attention of the vision encoder.
#include "ptx.cuh"
#include "seq_tile.cuh"
#include "tma_host.h"

namespace ne {

constexpr int kKernelFm = 27;
constexpr int kFmBlk = 64;                     // keys per block: one cache page
constexpr int kFmSlot = kFmBlk * 128;          // 64 rows x 64 bf16 columns
constexpr int kFmQ = 128 * 128;                // a chunk of Q: 128 rows x 64 columns
constexpr int kFmMaxSlots = 24;
constexpr int kFmGroups = 32;                  // barriers of groups in flight; a group has at least one slot

struct FmArgs {
  const int* block_tables; int bt_stride;      // paged
  const int* cu_seqlens_q; const int* context_lens; int num_seqs;      // context_lens null: the keys are the sequence's own tokens
  int T, Hq, g, tq, tiles, splits;             // tq tokens per tile of g tq rows, up to `tiles` tiles per CTA
  int nc, nv, ksteps, npv, dv;                 // 64-column chunks of K and V, K = 16 steps of the first product, N of the second, value columns
  int rope_chunk;                              // chunks of K from this one on come from the rotary map, shared by the heads
  int slots, window, causal, paged;
  uint32_t tmem_cols;
  float scale_log2;
  __nv_bfloat16* out;                          // [T, Hq, dv]
  float* part; float* lse2;                    // [splits, T, Hq, dv], [splits, T, Hq] (splits > 1)
  // the operands again, for rows that are taken once more on the CUDA cores: k rows k_dim wide, then those of the rotary map up to d; heads k_dim / dv apart
  const __nv_bfloat16* q; const __nv_bfloat16* k; const __nv_bfloat16* v; const __nv_bfloat16* k_rope;
  long long q_ld, k_ld, v_ld, r_ld;            // k_ld, v_ld: from one token to the next (pages too)
  int d, k_dim;
};

// (x, y) <- (x, y) scale + shift, and sum += (x, y): two fp32 operations in one instruction
__device__ __forceinline__ void fma2(uint32_t& x, uint32_t& y, float scale, float shift) {
  asm("{\n .reg .b64 a, b, c;\n mov.b64 a, {%0, %1};\n mov.b64 b, {%2, %2};\n mov.b64 c, {%3, %3};\n fma.rn.ftz.f32x2 a, a, b, c;\n mov.b64 {%0, %1}, a;\n}"
      : "+r"(x), "+r"(y) : "f"(scale), "f"(shift));
}
__device__ __forceinline__ void add2(float (&sum)[2], uint32_t x, uint32_t y) {
  asm("{\n .reg .b64 a, b;\n mov.b64 a, {%0, %1};\n mov.b64 b, {%2, %3};\n add.rn.ftz.f32x2 a, a, b;\n mov.b64 {%0, %1}, a;\n}" : "+f"(sum[0]), "+f"(sum[1]) : "r"(x), "r"(y));
}
__device__ __forceinline__ uint32_t ex2(uint32_t x) {
  asm volatile("ex2.approx.ftz.f32 %0, %0;" : "+r"(x));      // volatile: in this order, back to back
  return x;
}

__device__ __forceinline__ void mbar_test3(uint32_t a, uint32_t pa, uint32_t b, uint32_t pb, uint32_t c, uint32_t pc, bool& ra, bool& rb, bool& rc) {
  uint32_t x, y, z;
  asm volatile("{\n .reg .pred p, q, r;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%3], %4;\n mbarrier.test_wait.parity.shared::cta.b64 q, [%5], %6;\n"
               " mbarrier.test_wait.parity.shared::cta.b64 r, [%7], %8;\n selp.u32 %0, 1, 0, p;\n selp.u32 %1, 1, 0, q;\n selp.u32 %2, 1, 0, r;\n}\n"
               : "=r"(x), "=r"(y), "=r"(z) : "r"(a), "r"(pa), "r"(b), "r"(pb), "r"(c), "r"(pc) : "memory");
  ra = x; rb = y; rc = z;
}

// tokens of a sequence; those past the tensors' end are none of its rows (n_tok), nor keys where they are the tokens themselves
__device__ __forceinline__ int fm_len(const FmArgs& a, int seq, int beg) { return (a.context_lens ? a.cu_seqlens_q[seq + 1] : min(a.cu_seqlens_q[seq + 1], a.T)) - beg; }

// sum of a[i] b[i], n a multiple of 8, both on 16-byte boundaries
__device__ __forceinline__ float fm_dot(const __nv_bfloat16* a, const __nv_bfloat16* b, int n) {
  float s = 0.f;
#pragma unroll 1
  for (int i = 0; i < n; i += 8) {
    const uint4 x = *reinterpret_cast<const uint4*>(a + i), y = *reinterpret_cast<const uint4*>(b + i);
    const uint32_t wx[4] = {x.x, x.y, x.z, x.w}, wy[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
    for (int e = 0; e < 4; e++) {
      const float2 f = unpack_bf16x2(wx[e]), g = unpack_bf16x2(wy[e]);
      s = fmaf(f.x, g.x, fmaf(f.y, g.y, s));
    }
  }
  return s;
}

// One row once more, by a warp on the CUDA cores: keys [lo, hi] of the sequence's page table `bt` (or its own tokens, k_beg on).  A tile's products multiply every
// value row that one of its rows sees; zero times an infinity, or no number, among those that others may not see reaches them, an infinity's two terms may have
// opposite signs, and a sum may overflow before it is divided.  So a row whose sums are not all finite is taken again, values of probability zero left out.  m, inv:
// reference exponent and 1 / sum of the row, which come from scores alone and stand (inv 0: no key).  Never reached with finite values, and rolled up, so that it
// costs the loops of the kernel no register (107 -> 106; as a call, or at the end for all warps, it cost 2 % of the MLA prompts' time, so nothing).
template <bool kSplitP>
__device__ __forceinline__ void fmha_row_again(const FmArgs& a, const int* bt, int k_beg, int hkv, long long tok, int head, int lo, int hi, float m, float inv, int split) {
  const int lane = (int)lane_id();
  const __nv_bfloat16* q = a.q + tok * a.q_ld + (long long)head * a.d;
  float acc[8];                              // columns 64 i + 2 lane and the next
#pragma unroll
  for (int i = 0; i < 8; i++) acc[i] = 0.f;
  auto token = [&](int key) -> long long {   // row of the key, -1: of a page that is none
    if (!a.paged) return k_beg + key;
    const int page = bt[key / kFmBlk];
    return NE_INDEX_OK(page, BK_CACHE_PAGES, kKernelFm, __LINE__) ? (long long)page * kFmBlk + key % kFmBlk : -1;
  };
#pragma unroll 1
  for (int key0 = inv > 0.f ? lo : hi + 1; key0 <= hi; key0 += 32) {
    const long long row = key0 + lane <= hi ? token(key0 + lane) : -1;
    float w = 0.f;
    if (row >= 0) {
      float s = fm_dot(q, a.k + row * a.k_ld + (long long)hkv * a.k_dim, a.k_dim);
      if (a.k_dim < a.d) s += fm_dot(q + a.k_dim, a.k_rope + row * a.r_ld, a.d - a.k_dim);
      w = exp2f(fmaf(s, a.scale_log2, -m));
      if (!kSplitP) w = __bfloat162float(__float2bfloat16(w));
      w *= inv;
    }
#pragma unroll 1
    for (int e = 0; e < 32; e++) {
      const float we = __shfl_sync(0xffffffffu, w, e);
      const long long re = __shfl_sync(0xffffffffu, row, e);
      if (we == 0.f) continue;
      const __nv_bfloat16* v = a.v + re * a.v_ld + (long long)hkv * a.dv;
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const int c = 64 * i + 2 * lane;
        if (c < a.dv) {
          const float2 f = unpack_bf16x2(*reinterpret_cast<const uint32_t*>(v + c));
          acc[2 * i] = fmaf(we, f.x, acc[2 * i]); acc[2 * i + 1] = fmaf(we, f.y, acc[2 * i + 1]);
        }
      }
    }
  }
  const long long orow = tok * a.Hq + head;
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const int c = 64 * i + 2 * lane;
    if (c >= a.dv) continue;
    if (a.splits == 1) *reinterpret_cast<uint32_t*>(a.out + orow * a.dv + c) = pack_bf16x2(acc[2 * i], acc[2 * i + 1]);
    else *reinterpret_cast<float2*>(a.part + ((long long)split * a.T * a.Hq + orow) * a.dv + c) = make_float2(acc[2 * i], acc[2 * i + 1]);
  }
}

// Those of a softmax warp's rows that `again` names: lanes hold their rows' m and inv.  The geometry is worked out anew: nothing of this is alive in the loops.
template <bool kSplitP>
__device__ __forceinline__ void fmha_rows_again(const FmArgs& a, unsigned again, int seq, int tok0, int row0, float m, float inv) {
  const int hkv = blockIdx.y, split = blockIdx.z, q_beg = a.cu_seqlens_q[seq], q_len = fm_len(a, seq, q_beg), ctx = a.context_lens ? a.context_lens[seq] : q_len;
  const int n_tok = min(a.tq * a.tiles, min(q_beg + q_len, a.T) - tok0), base_limit = a.causal ? ctx - q_len + (tok0 - q_beg) : ctx - 1;
  const int vis_hi = a.causal ? base_limit + n_tok - 1 : base_limit, vis_lo = a.window > 0 ? max(0, base_limit - a.window + 1) : 0;
  const int first = vis_lo / kFmBlk, total = vis_hi >= 0 ? vis_hi / kFmBlk + 1 - first : 0, per_split = (total + a.splits - 1) / a.splits;
  const int key_lo = (first + split * per_split) * kFmBlk, key_hi = (first + min(total, (split + 1) * per_split)) * kFmBlk - 1;
#pragma unroll 1
  for (; again; again &= again - 1) {
    const int l = __ffs(again) - 1, row = row0 + l, tl = (row >> 7) * a.tq + (row & 127) / a.g, limit = a.causal ? base_limit + tl : base_limit;
    fmha_row_again<kSplitP>(a, a.paged ? a.block_tables + (long long)seq * a.bt_stride : nullptr, q_beg, hkv, tok0 + tl, hkv * a.g + (row & 127) % a.g,
                            max(key_lo, a.window > 0 ? limit - a.window + 1 : 0), min(key_hi, limit), __shfl_sync(0xffffffffu, m, l), __shfl_sync(0xffffffffu, inv, l), split);
  }
}

// kWG: softmax warpgroups = most tiles per CTA; kSlots: score slots of a tile
template <int kWG, bool kSplitP, int kSlots>
__global__ void __launch_bounds__(128 + 128 * kWG, kWG == 1 && kSlots == 2 ? 2 : 1)
fmha_kernel(const __grid_constant__ CUtensorMap q_map, const __grid_constant__ CUtensorMap k_map, const __grid_constant__ CUtensorMap v_map,
            const __grid_constant__ CUtensorMap r_map, const __grid_constant__ FmArgs a) {
  pdl_wait();                     // dependent launch: nothing above this line touches global memory
  extern __shared__ uint8_t smem_raw[];
  // swizzled tiles need 1024-byte alignment; behind static shared memory the dynamic part starts on a 16-byte boundary
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem;                                    // [tile][chunk][128 rows x 128 B]
  uint8_t* sKV = sQ + kWG * a.nc * kFmQ;
  __shared__ uint64_t bars[2 * kFmGroups + 5 + 3 * kWG * kSlots];
  __shared__ uint32_t s_tmem;
  __shared__ int s_abort, s_seq, s_tok;
  volatile int* abort_flag = &s_abort;
  // scores, probabilities, products: [tile][slot]
  constexpr int kBars = 8 * kWG * kSlots;
  const uint32_t b_full = smem_u32(bars), b_empty = b_full + 8 * kFmGroups, b_q = b_empty + 8 * kFmGroups, b_s = b_q + 8, b_p = b_s + kBars, b_pv = b_p + kBars,
                 b_go = b_pv + kBars, b_fix = b_go + 16;
  auto slot_of = [](int j) { return kSlots == 2 ? j & 1 : j % kSlots; };
  auto phase_of = [](int j) { return (uint32_t)(j / kSlots) & 1; };
  const int warp = threadIdx.x >> 5;
  const int hkv = blockIdx.y, split = blockIdx.z;
  if (warp == 0) {
    int seq, tok;
    // later tiles of a sequence see more keys: they start first
    find_seq_tile(a.cu_seqlens_q, a.num_seqs, a.tq * a.tiles, (int)(gridDim.x - 1 - blockIdx.x), seq, tok);
    if (lane_id() == 0) { s_seq = seq; s_tok = tok; }
  }
  if (warp == 2) { tmem_alloc(smem_u32(&s_tmem), a.tmem_cols); tmem_relinquish(); }
  __syncthreads();
  const int seq = s_seq, tok0 = s_tok;

  // geometry (uniform over the CTA)
  int nt = 1, nblk = 0, blk0 = 0, n_tok = 0, base_limit = -1, vis_lo = 0, vis_hi = -1, k_beg = 0;
  if (seq >= 0) {
    const int q_beg = a.cu_seqlens_q[seq], q_len = fm_len(a, seq, q_beg), ctx = a.context_lens ? a.context_lens[seq] : q_len;
    n_tok = min(a.tq * a.tiles, min(q_beg + q_len, a.T) - tok0);
    nt = n_tok > a.tq ? 2 : 1;
    k_beg = q_beg;
    base_limit = a.causal ? ctx - q_len + (tok0 - q_beg) : ctx - 1;          // last key visible to the tile's first token
    vis_hi = a.causal ? base_limit + n_tok - 1 : base_limit;                  // ... to any of its tokens
    vis_lo = a.window > 0 ? max(0, base_limit - a.window + 1) : 0;
    const int first = vis_lo / kFmBlk, total = vis_hi >= 0 ? vis_hi / kFmBlk + 1 - first : 0;
    const int per_split = (total + a.splits - 1) / a.splits;
    blk0 = first + split * per_split;
    nblk = max(0, min(total, (split + 1) * per_split) - split * per_split);
  }
  if (threadIdx.x == 32) {
    for (int i = 0; i < kFmGroups; i++) { mbar_init(b_full + 8 * i, 1); mbar_init(b_empty + 8 * i, nt); }
    mbar_init(b_q, 1);
    for (int i = 0; i < kWG * kSlots; i++) { mbar_init(b_s + 8 * i, 1); mbar_init(b_p + 8 * i, 4); mbar_init(b_pv + 8 * i, 1); }
    for (int i = 0; i < 2; i++) { mbar_init(b_go + 8 * i, 1); mbar_init(b_fix + 8 * i, 32); }
    s_abort = 0;
    mbar_fence_init();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_trigger();                  // behind the TMEM allocation: a CTA of the next grid never holds columns this grid waits for
  constexpr uint32_t kO = kSlots == 2 ? 128 * kWG : 256;
  const uint32_t tmem = s_tmem;   // S/P of tile t, block j at columns 128 t + 64 slot(j), O of tile t behind them at kO + 128 t
  const bool fix_lo = nblk > 0 && blk0 * kFmBlk < vis_lo, fix_hi = nblk > 0 && (blk0 + nblk) * kFmBlk - 1 > vis_hi;

  if (warp == 0) {
    if (nblk > 0 && elect_one()) {
      mbar_expect_tx(b_q, nt * a.nc * a.g * a.tq * 128);
      for (int t = 0; t < nt; t++)
        for (int c = 0; c < a.nc; c++) tma_load_3d(smem_u32(sQ + (t * a.nc + c) * kFmQ), &q_map, b_q, c * 64, hkv * a.g, tok0 + t * a.tq);
      int s = 0, group = 0, tail = 0, room = a.slots;      // groups are released in the order of loading
      auto size_of = [&](int g) { return g == 2 * nblk - 1 || (g > 0 && !(g & 1)) ? a.nv : a.nc; };      // K K V K V .. K V V
      const int* bt = a.block_tables + (long long)seq * a.bt_stride;
      auto load = [&](int j, bool v) -> bool {
        const int key0 = (blk0 + j) * kFmBlk;
        int page = 0;
        if (a.paged) {
          page = bt[blk0 + j];
          if (!NE_INDEX_OK(page, BK_CACHE_PAGES, kKernelFm, __LINE__)) page = 0;
        }
        const int n = v ? a.nv : a.nc;
        for (; room < n; tail++) {
          if (!mbar_wait(b_empty + 8 * (tail % kFmGroups), (tail / kFmGroups) & 1, abort_flag, kKernelFm, 100)) return false;
          room += size_of(tail);
        }
        room -= n;
        const uint32_t bar = b_full + 8 * (group++ % kFmGroups);
        mbar_expect_tx(bar, n * kFmSlot);
        for (int c = 0; c < n; c++) {
          const uint32_t dst = smem_u32(sKV + s * kFmSlot);
          if (a.paged) {
            tma_load_4d(dst, v ? &v_map : &k_map, bar, c * 64, hkv, 0, page);
          } else if (!v && c >= a.rope_chunk) {
            tma_load_2d(dst, &r_map, bar, (c - a.rope_chunk) * 64, k_beg + key0);
          } else {
            tma_load_3d(dst, v ? &v_map : &k_map, bar, c * 64, hkv, k_beg + key0);      // rows past the tensor's end are zero-filled
          }
          if (++s == a.slots) s = 0;
        }
        if (v && j == 0 && fix_lo) mbar_arrive(b_go);
        if (v && j == nblk - 1 && fix_hi) mbar_arrive(b_go + 8);
        return true;
      };
      bool ok = load(0, false);
      if (ok && nblk > 1) ok = load(1, false);
      for (int j = 0; ok && j < nblk; j++) ok = load(j, true) && (j + 2 >= nblk || load(j + 2, false));
    }
  } else if (warp <= 2) {
    const int t = warp - 1;       // the issuer's tile
    if (t < nt && nblk > 0 && elect_one()) {
      constexpr uint32_t kIdS = make_idesc(FMT_BF16, FMT_BF16, 128, kFmBlk);
      const uint32_t id_pv = make_idesc(FMT_BF16, FMT_BF16, 128, (uint32_t)a.npv, 0, 1);      // B (= V) is MN-major
      // descriptors of the operands' first tiles; others by adding their distance (in units of 16 bytes)
      constexpr uint32_t kTile = kFmSlot >> 4;
      const uint64_t dq = make_smem_desc(smem_u32(sQ), 16, 1024, SW_128B) + t * a.nc * (kFmQ >> 4), dk = make_smem_desc(smem_u32(sKV), 16, 1024, SW_128B),
                     dv = make_smem_desc(smem_u32(sKV), kFmSlot, 1024, SW_128B);
      const uint32_t o = tmem + kO + t * 128, s0 = tmem + t * 128, bs = b_s + 8 * kSlots * t, bp = b_p + 8 * kSlots * t, bpv = b_pv + 8 * kSlots * t;
      // groups in the order of loading: number and first slot of the next one (no division: its reciprocal would wait behind the softmax's exponentials)
      int s = 0, group = 0;
      auto full = [&](int g) { return b_full + 8 * (g % kFmGroups); };
      auto parity = [](int g) { return (uint32_t)(g / kFmGroups) & 1; };
      auto step = [&](int n, int& first, uint32_t& done) {
        first = s; done = b_empty + 8 * (group++ % kFmGroups);
        s += n;
        if (s >= a.slots) s -= a.slots;
      };
      int k0 = 0, v0 = 0;
      uint32_t kd = 0, vd = 0;
      bool split_before = false;
      auto scores = [&](int j) {
        tc_fence_after();
        const uint32_t d = s0 + slot_of(j) * kFmBlk;
        int ks = k0;
        for (int c = 0; c < a.nc; c++) {
          const uint64_t qa = dq + c * (kFmQ >> 4), ka = dk + ks * kTile;
          const int steps = a.ksteps - 4 * c;
          umma_f16(d, qa, ka, kIdS, c != 0);
          if (steps > 1) umma_f16(d, qa + 2, ka + 2, kIdS, 1);
          if (steps > 2) umma_f16(d, qa + 4, ka + 4, kIdS, 1);
          if (steps > 3) umma_f16(d, qa + 6, ka + 6, kIdS, 1);
          if (++ks == a.slots) ks = 0;
        }
        tc_commit(bs + 8 * slot_of(j));
        tc_commit(kd);
      };
      bool ok = mbar_wait(b_q, 0, abort_flag, kKernelFm, 200);
      for (int j = 0; ok && j < 2 && j < nblk; j++) {
        ok = mbar_wait(full(group), parity(group), abort_flag, kKernelFm, 210);
        step(a.nc, k0, kd);
        if (ok) scores(j);
      }
      for (int j = 0; ok && j < nblk; j++) {
        const bool next = j + 2 < nblk;
        const uint32_t bj = bp + 8 * slot_of(j), pp = phase_of(j);
        const uint32_t bv = full(group), pv = parity(group), bk = next ? full(group + 1) : bv, pk = next ? parity(group + 1) : pv;
        bool rv, rk, rp;
        mbar_test3(bv, pv, bk, pk, bj, pp, rv, rk, rp);      // three tests for the price of one
        if (!rv) ok = mbar_wait(bv, pv, abort_flag, kKernelFm, 220);
        if (ok && !rk) ok = mbar_wait(bk, pk, abort_flag, kKernelFm, 212);
        if (ok && j == 0 && fix_lo) ok = mbar_wait(b_fix, 0, abort_flag, kKernelFm, 221);
        if (ok && j == nblk - 1 && fix_hi) ok = mbar_wait(b_fix + 8, 0, abort_flag, kKernelFm, 222);
        if (ok && !rp) ok = mbar_wait(bj, pp, abort_flag, kKernelFm, 230);
        step(a.nv, v0, vd);
        if (next) step(a.nc, k0, kd);
        const int head = min(a.nv, a.slots - v0);
        // products of other column ranges than those of the block before add to the same O: behind them
        if (ok && kSlots == 3 && j > 0 && (head != a.nv || split_before)) ok = mbar_wait(bpv + 8 * slot_of(j - 1), phase_of(j - 1), abort_flag, kKernelFm, 242);
        split_before = head != a.nv;
        if (!ok) break;
        tc_fence_after();
        const uint32_t p = s0 + slot_of(j) * kFmBlk;
        // the chunks of V lie in consecutive ring slots; where they wrap around the ring's end, the product is issued in two column ranges
        const uint64_t va = dv + v0 * kTile;
        if (head == a.nv) {
#pragma unroll
          for (int x = 0; x < (kSplitP ? 2 : 1); x++)
#pragma unroll
            for (int ks = 0; ks < 4; ks++) umma_f16_ts(o, p + x * 32 + ks * 8, va + ks * 128, id_pv, (x | ks) ? 1u : (uint32_t)(j != 0));
        } else {
          const uint32_t id_a = make_idesc(FMT_BF16, FMT_BF16, 128, (uint32_t)head * 64, 0, 1), id_b = make_idesc(FMT_BF16, FMT_BF16, 128, (uint32_t)(a.npv - head * 64), 0, 1);
#pragma unroll
          for (int x = 0; x < (kSplitP ? 2 : 1); x++)
#pragma unroll
            for (int ks = 0; ks < 4; ks++) {
              umma_f16_ts(o, p + x * 32 + ks * 8, va + ks * 128, id_a, (x | ks) ? 1u : (uint32_t)(j != 0));
              umma_f16_ts(o + head * 64, p + x * 32 + ks * 8, dv + ks * 128, id_b, (x | ks) ? 1u : (uint32_t)(j != 0));
            }
        }
        tc_commit(bpv + 8 * slot_of(j));
        tc_commit(vd);
        // the products whose probabilities lie in the next scores' slot; with two slots these very ones, which also orders them before the next products
        if (kSlots == 2 ? j + 1 < nblk : next && j > 0) ok = mbar_wait(bpv + 8 * slot_of(j - (kSlots - 2)), phase_of(j - (kSlots - 2)), abort_flag, kKernelFm, 241, 0);
        if (ok && next) scores(j + 2);
      }
    }
  } else if (warp < 4) {
    for (int w = 0; w < 2; w++) {
      if (!(w ? fix_hi : fix_lo)) continue;
      const int j = w ? nblk - 1 : 0, key0 = (blk0 + j) * kFmBlk;
      // group and first slot of the block's V in the order of loading
      const int g = min(j + 2, nblk) + j, p0 = min(j + 2, nblk) * a.nc + j * a.nv;
      // once its loads are under way the phase waited for is the current one
      if (mbar_wait(b_go + 8 * w, 0, abort_flag, kKernelFm, 400) && mbar_wait(b_full + 8 * (g % kFmGroups), (g / kFmGroups) & 1, abort_flag, kKernelFm, 410))
        for (int i = (int)lane_id(); i < a.nv * kFmBlk; i += 32) {
          const int key = key0 + (i & (kFmBlk - 1));
          if (w ? key > vis_hi : key < vis_lo) {
            uint4* dst = reinterpret_cast<uint4*>(sKV + ((p0 + i / kFmBlk) % a.slots) * kFmSlot + (i & (kFmBlk - 1)) * 128);
#pragma unroll
            for (int x = 0; x < 8; x++) dst[x] = make_uint4(0, 0, 0, 0);
          }
        }
      fence_proxy_async_smem();
      mbar_arrive(b_fix + 8 * w);
    }
  } else {
    const int t = (warp - 4) >> 2, wq = warp & 3, row = wq * 32 + (int)lane_id();
    const uint32_t lane_addr = (uint32_t)(wq * 32) << 16;
    const int tl = t * a.tq + row / a.g, head = hkv * a.g + row % a.g;        // token of the CTA's tiles
    const bool row_ok = row < a.g * a.tq && tl < n_tok;
    const int limit = row_ok ? (a.causal ? base_limit + tl : base_limit) : -1;
    const int lowest = a.window > 0 ? limit - a.window + 1 : 0;
    const uint32_t tmem_o = tmem + kO + t * 128 + lane_addr;
    float m_run = -INFINITY, l_run = 0.f;
    bool ok = true;
    int last = -1;
    const int own = t < nt ? nblk : 0;
    const uint32_t bs = b_s + 8 * kSlots * t, bp = b_p + 8 * kSlots * t, bpv = b_pv + 8 * kSlots * t;
    bool ready = false;
    for (int j = 0; ok && j < own; j++) {
      const int key0 = (blk0 + j) * kFmBlk;
      const uint32_t ts = tmem + t * 128 + slot_of(j) * kFmBlk + lane_addr;
      if (!ready && !mbar_wait(bs + 8 * slot_of(j), phase_of(j), abort_flag, kKernelFm, 300)) { ok = false; break; }
      tc_fence_after();
      __syncwarp();
      uint32_t r[64];
      tmem_ld_32x32b_x32(ts, *reinterpret_cast<uint32_t(*)[32]>(r));
      tmem_ld_32x32b_x32(ts + 32, *reinterpret_cast<uint32_t(*)[32]>(r + 32));
      tc_wait_ld();
      if (key0 + kFmBlk - 1 > limit || key0 < lowest) {
#pragma unroll
        for (int i = 0; i < 64; i++)
          if (key0 + i > limit || key0 + i < lowest) r[i] = 0xff800000u;
      }
#ifdef NE_DEBUG_BOUNDS
      if (a.paged && !NE_INDEX_OK(a.block_tables[(long long)seq * a.bt_stride + blk0 + j], BK_CACHE_PAGES, kKernelFm, __LINE__)) {      // keys of a page that is none
#pragma unroll
        for (int i = 0; i < 64; i++) r[i] = 0xff800000u;
      }
#endif
      float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int i = 0; i < 64; i += 8)
#pragma unroll
        for (int e = 0; e < 4; e++) mx[e] = fmaxf(mx[e], fmaxf(__uint_as_float(r[i + 2 * e]), __uint_as_float(r[i + 2 * e + 1])));
      float m_tile = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * a.scale_log2;
      // 32-bit probabilities: the reference is a whole power of two, so rescaling by it is exact and the two terms of a probability are the same whatever the
      // slices and blocks are.  bf16 probabilities: the largest one is exactly 1, and a row that looks at few keys has the smaller error.
      if (kSplitP) m_tile = ceilf(m_tile);
      // lazy rescaling: the reference maximum only moves when the block's maximum exceeds it by more than 2^8
      const bool first_valid = m_run == -INFINITY;
      const float m_new = (first_valid || m_tile > m_run + 8.f) ? fmaxf(m_run, m_tile) : m_run;
      const float alpha = (m_new == -INFINITY || first_valid) ? 1.f : exp2f(m_run - m_new);
      const float neg_m = (m_new == -INFINITY) ? 0.f : -m_new;
      float ps[2] = {0.f, 0.f};
      __syncwarp();                          // rows at a limit took a branch of their own
      // 32 columns at a time; the next ones' exponentials are under way while these are packed and stored
      auto exps = [&](int c) {
#pragma unroll
        for (int j = 0; j < 16; j++) fma2(r[c * 32 + 2 * j], r[c * 32 + 2 * j + 1], a.scale_log2, neg_m);
#pragma unroll
        for (int j = 0; j < 32; j++) r[c * 32 + j] = ex2(r[c * 32 + j]);
      };
      exps(0);
#pragma unroll
      for (int c = 0; c < 2; c++) {
        if (c < 1) exps(c + 1);
        uint32_t* x = r + c * 32;
        uint32_t hi[16];
        if constexpr (kSplitP) {
          uint32_t lo[16];
#pragma unroll
          for (int j = 0; j < 16; j++) {
            hi[j] = pack_bf16x2(__uint_as_float(x[2 * j]), __uint_as_float(x[2 * j + 1]));
            add2(ps, x[2 * j], x[2 * j + 1]);
            lo[j] = pack_bf16x2(__uint_as_float(x[2 * j]) - __uint_as_float(hi[j] << 16), __uint_as_float(x[2 * j + 1]) - __uint_as_float(hi[j] & 0xffff0000u));
          }
          tmem_st_32x32b_x16(ts + 32 + c * 16, lo);
        } else {
#pragma unroll
          for (int j = 0; j < 16; j++) {       // sum what the product will see, so numerator and denominator stay consistent
            hi[j] = pack_bf16x2(__uint_as_float(x[2 * j]), __uint_as_float(x[2 * j + 1]));
            add2(ps, hi[j] << 16, hi[j] & 0xffff0000u);
          }
        }
        tmem_st_32x32b_x16(ts + c * 16, hi);
      }
      __syncwarp();
      ready = j + 1 < own && mbar_test(bs + 8 * slot_of(j + 1), phase_of(j + 1));
      l_run = l_run * alpha + (ps[0] + ps[1]);
      m_run = m_new;
      if (last >= 0 && __any_sync(0xffffffffu, alpha < 1.f)) {
        if (!mbar_wait(bpv + 8 * slot_of(last), phase_of(last), abort_flag, kKernelFm, 310)) { ok = false; break; }
        tc_fence_after();
#pragma unroll 1
        for (int cblk = 0; cblk < (a.npv + 15) / 16; cblk++) {
          uint32_t o[16];
          tmem_ld_32x32b_x16(tmem_o + cblk * 16, o);
          tc_wait_ld();
#pragma unroll
          for (int j = 0; j < 16; j++) o[j] = __float_as_uint(__uint_as_float(o[j]) * alpha);
          tmem_st_32x32b_x16(tmem_o + cblk * 16, o);
        }
      }
      tc_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane_id() == 0) mbar_arrive(bp + 8 * slot_of(j));
      last = j;
    }
    if (ok && last >= 0) ok = mbar_wait(bpv + 8 * slot_of(last), phase_of(last), abort_flag, kKernelFm, 320);
    const bool have = ok && last >= 0;
    const long long rows = (long long)a.T * a.Hq, orow = row_ok ? (long long)(tok0 + tl) * a.Hq + head : 0;
    if (have) tc_fence_after();
    __syncwarp();
    const float inv = have && l_run > 0.f ? 1.f / l_run : 0.f;
    float all[2] = {0.f, 0.f};               // no finite number if one of the row's sums is none
#pragma unroll 1
    for (int cblk = 0; cblk < (a.npv + 15) / 16; cblk++) {
      uint32_t o[16];
      __syncwarp();                          // the lanes of rows outside the tile skip the stores below
      if (have) {
        tmem_ld_32x32b_x16(tmem_o + cblk * 16, o);
        tc_wait_ld();
#pragma unroll
        for (int j = 0; j < 16; j += 2) add2(all, o[j], o[j + 1]);
#pragma unroll
        for (int j = 0; j < 16; j++) o[j] = __float_as_uint(__uint_as_float(o[j]) * inv);
      } else {
#pragma unroll
        for (int j = 0; j < 16; j++) o[j] = 0u;
      }
      if (!row_ok) continue;
#pragma unroll
      for (int v = 0; v < 2; v++) {          // dv is a multiple of 8
        const int col = cblk * 16 + v * 8;
        if (col >= a.dv) continue;
        const float* f = reinterpret_cast<const float*>(o + v * 8);
        if (a.splits == 1) {
          *reinterpret_cast<uint4*>(a.out + orow * a.dv + col) = make_uint4(pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3]), pack_bf16x2(f[4], f[5]), pack_bf16x2(f[6], f[7]));
        } else {
          float* dst = a.part + ((long long)split * rows + orow) * a.dv + col;
          *reinterpret_cast<float4*>(dst) = make_float4(f[0], f[1], f[2], f[3]);
          *reinterpret_cast<float4*>(dst + 4) = make_float4(f[4], f[5], f[6], f[7]);
        }
      }
    }
    // rows with infinities or no numbers among their sums, whose scores are numbers
    const unsigned again = __ballot_sync(0xffffffffu, row_ok && !(fabsf(all[0] + all[1]) < INFINITY) && l_run >= 0.f && l_run < INFINITY);
    if (again) fmha_rows_again<kSplitP>(a, again, seq, tok0, t * 128 + wq * 32, m_run, inv);
    if (a.splits > 1 && row_ok) a.lse2[(long long)split * rows + orow] = (have && l_run != 0.f) ? m_run + log2f(l_run) : -INFINITY;      // no number: the merge passes it on
  }

  tc_fence_before();
  __syncthreads();
  if (*abort_flag && threadIdx.x == 0) for (int i = 0; i < 2000; i++) __nanosleep(1000);      // copies in flight
  __syncthreads();
  if (warp == 2) { tc_fence_after(); tmem_dealloc(tmem, a.tmem_cols); }
}

constexpr int kFmSmem = 232448 - 1024;         // dynamic shared memory limit of a block less the static part
constexpr int kFmSmemHalf = 233472 / 2 - 2 * 1024;      // where two blocks share an SM (1 KB of each is the system's)

template <int kWG, bool kSplitP, int kSlots>
static int fmha_launch(const CUtensorMap& q, const CUtensorMap& k, const CUtensorMap& v, const CUtensorMap& r, const FmArgs& a, int grid_x, int heads, cudaStream_t st) {
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(fmha_kernel<kWG, kSplitP, kSlots>, cudaFuncAttributeMaxDynamicSharedMemorySize, kFmSmem);
    if (e != cudaSuccess) return (int)e;
    configured = true;
  }
  return (int)launch_pdl(fmha_kernel<kWG, kSplitP, kSlots>, dim3((unsigned)grid_x, (unsigned)heads, (unsigned)a.splits), dim3(128 + 128 * kWG),
                         (size_t)kWG * a.nc * kFmQ + (size_t)a.slots * kFmSlot + 1024, st, q, k, v, r, a);
}

}  // namespace ne

using namespace ne;

// q [T, Hq, D] with row stride q_ld (elements; heads D apart), keys / values either pages k, v [num_blocks, 64, Hkv, D or Dv] contiguous (block_tables
// not null) or rows [T, Hkv, D or Dv] with row strides k_ld, v_ld; k_rope not null (ragged only): the last D - Dk_nope columns of every head's key are the
// row k_rope [T, D - Dk_nope] (row stride r_ld), k_nope heads k_head apart.  context_lens null: keys are the sequence's own tokens.
// split_p: probabilities as two bf16 terms.  splits > 1: part / lse2 as ne_attn_merge takes them.
extern "C" int ne_fmha(const void* q, long long q_ld, const void* k, long long k_ld, int k_dim, const void* k_rope, long long r_ld, const void* v, long long v_ld,
                       int num_blocks, const int* block_tables, int bt_stride, const int* cu_seqlens_q, const int* context_lens, int num_seqs, int T, int Hq,
                       int Hkv, int D, int Dv, int tiles, int grid_x, int splits, int window, int causal, float scale, int split_p, void* out, float* part,
                       float* lse2, cudaStream_t st) {
  if (T <= 0) return 0;
  if (Hkv < 1 || Hq % Hkv || splits < 1 || (splits > 1 && (!part || !lse2)) || grid_x < 1 || Hkv > 65535) return 1001;
  if (Hq / Hkv > 128 || D < 8 || D > 256 || D % 8 || Dv < 8 || Dv > 256 || Dv % 8 || tiles < 1 || tiles > (Dv <= 128 && D <= 192 ? 2 : 1)) return 1002;
  if (q_ld % 8 || q_ld < (long long)Hq * D || (block_tables == nullptr && (k_ld % 8 || v_ld % 8)) || (k_rope && (block_tables || r_ld % 8 || k_dim % 64 || k_dim >= D))) return 1003;
  FmArgs a;
  a.g = Hq / Hkv; a.tq = 128 / a.g; a.tiles = tiles; a.splits = splits; a.T = T; a.Hq = Hq;
  a.nc = (D + 63) / 64; a.nv = (Dv + 63) / 64; a.ksteps = (D + 15) / 16; a.npv = (Dv + 15) / 16 * 16; a.dv = Dv;
  a.rope_chunk = k_rope ? k_dim / 64 : a.nc;
  // single tiles: two CTAs share an SM where TMEM has room for both (one's loads and epilogue run beside the other's work)
  const bool share = tiles == 1 && Dv <= 128 && D <= 192;
  a.tmem_cols = share ? 256 : 512;
  a.slots = ((share ? kFmSmemHalf : kFmSmem) - 1024 - tiles * a.nc * kFmQ) / kFmSlot;
  if (a.slots > kFmMaxSlots) a.slots = kFmMaxSlots;
  if (a.slots < a.nc + a.nv) return 1004;                           // a block's K waits for its V, and the next block's K beside it
  a.window = window > 0 ? window : 0; a.causal = causal; a.paged = block_tables != nullptr;
  a.block_tables = block_tables; a.bt_stride = bt_stride; a.cu_seqlens_q = cu_seqlens_q; a.context_lens = context_lens; a.num_seqs = num_seqs;
  a.scale_log2 = scale * 1.4426950408889634f; a.out = (__nv_bfloat16*)out; a.part = part; a.lse2 = lse2;
  a.q = (const __nv_bfloat16*)q; a.k = (const __nv_bfloat16*)k; a.v = (const __nv_bfloat16*)v; a.k_rope = (const __nv_bfloat16*)k_rope;
  a.d = D; a.k_dim = k_rope ? k_dim : D; a.q_ld = q_ld; a.r_ld = r_ld; a.k_ld = a.paged ? (long long)Hkv * D : k_ld; a.v_ld = a.paged ? (long long)Hkv * Dv : v_ld;
  CUtensorMap mq, mk, mv, mr;
  {
    uint64_t dims[3] = {(uint64_t)D, (uint64_t)Hq, (uint64_t)T}, strides[2] = {(uint64_t)D * 2, (uint64_t)q_ld * 2};
    uint32_t box[3] = {64, (uint32_t)a.g, (uint32_t)a.tq};
    int rc = make_tmap(&mq, q, TMA_BF16, 3, dims, strides, box, TMA_SW_128); if (rc) return 2000 + rc;
  }
  for (int w = 0; w < 2; w++) {
    const uint64_t d = w ? Dv : (k_rope ? k_dim : D);
    int rc;
    if (a.paged) {
      uint64_t dims[4] = {d, (uint64_t)Hkv, 64, (uint64_t)num_blocks}, strides[3] = {d * 2, (uint64_t)Hkv * d * 2, 64 * (uint64_t)Hkv * d * 2};
      uint32_t box[4] = {64, 1, 64, 1};
      rc = make_tmap(w ? &mv : &mk, w ? v : k, TMA_BF16, 4, dims, strides, box, TMA_SW_128);
    } else {
      uint64_t dims[3] = {d, (uint64_t)Hkv, (uint64_t)T}, strides[2] = {d * 2, (uint64_t)(w ? v_ld : k_ld) * 2};
      uint32_t box[3] = {64, 1, kFmBlk};
      rc = make_tmap(w ? &mv : &mk, w ? v : k, TMA_BF16, 3, dims, strides, box, TMA_SW_128);
    }
    if (rc) return 2100 + rc;
  }
  mr = mk;
  if (k_rope) {
    uint64_t dims[2] = {(uint64_t)(D - k_dim), (uint64_t)T}, strides[1] = {(uint64_t)r_ld * 2};
    uint32_t box[2] = {64, kFmBlk};
    int rc = make_tmap(&mr, k_rope, TMA_BF16, 2, dims, strides, box, TMA_SW_128); if (rc) return 2200 + rc;
  }
  if (tiles == 2) return split_p ? fmha_launch<2, true, 2>(mq, mk, mv, mr, a, grid_x, Hkv, st) : fmha_launch<2, false, 2>(mq, mk, mv, mr, a, grid_x, Hkv, st);
  if (share) return split_p ? fmha_launch<1, true, 2>(mq, mk, mv, mr, a, grid_x, Hkv, st) : fmha_launch<1, false, 2>(mq, mk, mv, mr, a, grid_x, Hkv, st);
  return split_p ? fmha_launch<1, true, 3>(mq, mk, mv, mr, a, grid_x, Hkv, st) : fmha_launch<1, false, 3>(mq, mk, mv, mr, a, grid_x, Hkv, st);
}
