// Softmax attention for sm_100a on tcgen05 tensor cores, forward pass.
//
// One CTA per (batch, query head, pair of 128-query tiles); 640 threads:
//   warps 0..15 softmax: eight warps per query tile, two per 32 rows, one for each half of the key
//               tile's columns. A thread reads its 64 scores of S = Q·K^T from tensor memory
//               (tcgen05.ld), shares the row's maximum with the thread that holds the other half,
//               and writes P = exp2(S·scale - ref) (bf16) back over its own scores: the tensor
//               core takes P from tensor memory, so it crosses neither shared memory nor a proxy
//               fence. The per-row reference only moves when a row max outgrows it by 2^64 (then O
//               in tensor memory and the running sum are rescaled).
//   warp 16     TMA producer: both Q tiles once, then K and V tiles, two stages each (plain
//               TMA loads, no multicast).
//   warp 17     MMA issuer: S_x(j) = Q_x·K_j^T and O_x += P_x(j)·V_j, accumulated in
//               tensor memory; the two tiles' MMAs interleave so the tensor core works
//               on one tile while the other tile's softmax runs.
// GQA (H % G == 0), causal with bottom-right alignment, sliding window and attention
// sinks (one extra logit per head in the denominator) are handled in the mask / final
// normalisation. Fully masked key tiles are skipped. O leaves through shared memory (the tile's Q,
// no longer needed) and TMA stores.
//
// What bounds it: a tile's chain of S, softmax, P·V and the next S (S and P share tensor memory, all
// 512 columns are taken), against which the other tile's chain runs: 1024 cycles of tensor core and
// about 1900 of softmax per step, of which 1024 are the special-function unit's (16 ex2 per cycle and
// SM). What shortened it, 8 x 4096 tokens, 32/4 heads of 128 (776 TFLOP/s at first): P in tensor memory
// and two warps per scheduler and tile instead of one (888), P handed over in two parts so that the
// tensor core starts on the first while the second is worked on, the maximum in a pass of its own
// before them (1004). A third of the ex2 as polynomials on the FMA pipes was no gain (996): issue slots
// and tensor-memory latency, not that unit, fill the rest.
//
// Reference counterparts: cuDNN SDPA and FlashAttention-4 behind parallel/flash.py:573-678
// and parallel/fa4.py:410-573; the math is that of parallel/context.py:130 (xla).
#include "attention_sm100.h"
#include "common.cuh"
#include "gemm_sm100.h"

namespace bux {

constexpr int KID_ATTN_FWD = 2;
constexpr int QT = 128;  // query rows per CTA
constexpr int KT = 128;  // keys per tile
constexpr float LOG2E = 1.4426950408889634f;
constexpr float LN2 = 0.6931471805599453f;

struct AttnFwdParams {
  alignas(64) CUtensorMap tmap_q;
  alignas(64) CUtensorMap tmap_kv_k;
  alignas(64) CUtensorMap tmap_kv_v;
  alignas(64) CUtensorMap tmap_o;
  void* o; float* lse; const float* sinks; Status* status;
  const int* row_lo;  // [B, T] first visible key of each query (documents), or null
  int B, T, S, H, G;
  float scale_log2; int causal, window; bool by_length;
};

constexpr int FWD_SOFTMAX_WARPS = 16;
constexpr int FWD_THREADS = 32 * (FWD_SOFTMAX_WARPS + 4);   // + a warpgroup of the TMA warp, the MMA warp and two idle ones
// Five warps on a scheduler start with 96 registers each; the last warpgroup gives some of its own to
// the softmax warps, which spill with 96.
constexpr int FWD_LAUNCH_REGS = 96, FWD_SOFTMAX_REGS = 104, FWD_OTHER_REGS = 56;
static_assert(32 * FWD_SOFTMAX_WARPS * FWD_SOFTMAX_REGS + 128 * FWD_OTHER_REGS <= FWD_THREADS * FWD_LAUNCH_REGS,
              "a split above what the block was launched with would wait for ever");
constexpr float RESCALE_THRESHOLD = 64.f; // log2 units a row max may outgrow its reference

template <int D>
struct AttnFwdCfg {
  static constexpr int DC = D / 64;
  static constexpr int TILE_BYTES = DC * 16384;   // one [128 x D] bf16 tile
  static constexpr int ROW_BYTES = 6 * 128 * 2 * 4;  // row maxima (two buffers x two tiles x two halves), row sums
  static constexpr int SMEM_BYTES = TILE_BYTES * 6 + ROW_BYTES + 1024 + 256;
  static constexpr int TMEM_COLS = 512;           // S_A, S_B (128 each; P over them), O_A, O_B (D each)
};

// Two fp32 at once: a·b + c and a + b.
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("{\n.reg .b64 x, y, z;\nmov.b64 x, {%2, %3};\nmov.b64 y, {%4, %5};\nmov.b64 z, {%6, %7};\n"
      "fma.rn.f32x2 x, x, y, z;\nmov.b64 {%0, %1}, x;\n}\n"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return d;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  float2 d;
  asm("{\n.reg .b64 x, y;\nmov.b64 x, {%2, %3};\nmov.b64 y, {%4, %5};\nadd.rn.f32x2 x, x, y;\nmov.b64 {%0, %1}, x;\n}\n"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}
template <bool V> struct Flag { static constexpr bool value = V; };
__device__ __forceinline__ void pair_sync(int id) { asm volatile("bar.sync %0, 64;" ::"r"(id) : "memory"); }

template <int D>
__global__ void __launch_bounds__(FWD_THREADS, 1)
attn_fwd_kernel(const __grid_constant__ AttnFwdParams p) {
  using Cfg = AttnFwdCfg<D>;
  constexpr int DC = Cfg::DC;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem;                               // 2 tiles
  uint8_t* sK = sQ + 2 * Cfg::TILE_BYTES;           // 2 stages
  uint8_t* sV = sK + 2 * Cfg::TILE_BYTES;           // 2 stages
  float* row_max = reinterpret_cast<float*>(sV + 2 * Cfg::TILE_BYTES);  // [2 buffers][2 tiles][2 halves][128]
  float* row_sum = row_max + 2 * 2 * 2 * 128;                           // [2 tiles][2 halves][128]
  uint64_t* bars = reinterpret_cast<uint64_t*>(row_sum + 2 * 2 * 128);
  uint64_t* q_full = bars;
  uint64_t* k_full = bars + 1;     // [2]
  uint64_t* k_empty = bars + 3;    // [2]
  uint64_t* v_full = bars + 5;     // [2]
  uint64_t* v_empty = bars + 7;    // [2]
  uint64_t* s_full = bars + 9;     // [2] per query tile
  uint64_t* p_ready = bars + 11;   // [2] per query tile x [2] parts
  uint64_t* pv_full = bars + 15;   // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 17);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5;
  const int n_qt = (p.T + 2 * QT - 1) / (2 * QT);
  // the longest (latest) rows first under a causal mask, over every head of a chunk
  const AttnSlot slot = attn_slot(blockIdx.x, n_qt, p.H * p.B, p.by_length);
  const int qt = n_qt - 1 - slot.tile;
  const int h = slot.pair % p.H, b = slot.pair / p.H;
  const int g = h / (p.H / p.G);
  const int q0 = qt * 2 * QT;
  const int shift = p.S - p.T;
  const int s_tiles = (p.S + KT - 1) / KT;
  int lo[2], hi[2];
#pragma unroll
  for (int x = 0; x < 2; ++x) {
    const int qx = q0 + x * QT;
    hi[x] = s_tiles;
    if (p.causal) hi[x] = min(hi[x], (qx + QT - 1 + shift) / KT + 1);
    lo[x] = p.window > 0 ? max(0, (qx + shift - p.window + 1) / KT) : 0;
    // documents: the tile's first query has the earliest document start of the tile
    if (p.row_lo != nullptr && qx < p.T) lo[x] = max(lo[x], p.row_lo[(size_t)b * p.T + qx] / KT);
    if (qx >= p.T || hi[x] <= lo[x]) { lo[x] = 0; hi[x] = 0; }
  }
  const bool any0 = hi[0] > lo[0], any1 = hi[1] > lo[1];
  const int j_lo = any0 && any1 ? min(lo[0], lo[1]) : (any0 ? lo[0] : lo[1]);
  const int j_hi = max(hi[0], hi[1]);
  // With documents the second query tile may start seeing keys after the first one's last
  // key tile: the key tiles in between are seen by neither and are not loaded. Tiles that
  // are loaded are numbered 0, 1, ... (`slot_of`) for the stage rings and their parities.
  const int gap_at = (any0 && any1 && lo[1] > hi[0]) ? hi[0] : j_hi;
  const int gap = (any0 && any1 && lo[1] > hi[0]) ? lo[1] - hi[0] : 0;
  const int n_tiles = (any0 || any1) ? j_hi - j_lo - gap : 0;
  auto slot_of = [&](int j) { return j - j_lo - (j >= gap_at ? gap : 0); };
  auto tile_of = [&](int t) { return j_lo + t + (j_lo + t >= gap_at ? gap : 0); };
  Status* st = p.status;

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&k_full[i], 1); mbar_init(&k_empty[i], 1); mbar_init(&v_full[i], 1); mbar_init(&v_empty[i], 1);
      mbar_init(&s_full[i], 1); mbar_init(&p_ready[2 * i], 256); mbar_init(&p_ready[2 * i + 1], 256); mbar_init(&pv_full[i], 1);
    }
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 17) { tmem_alloc(tmem_slot, Cfg::TMEM_COLS); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp >= FWD_SOFTMAX_WARPS) reg_dec<FWD_OTHER_REGS>();
  if (warp == 16) {
    // -------------------------------------------------------------- TMA producer
    if (elect_one() && n_tiles > 0) {
      mbar_expect_tx(q_full, 2 * Cfg::TILE_BYTES);
      for (int x = 0; x < 2; ++x)
        for (int c = 0; c < DC; ++c)
          tma_load_2d(sQ + x * Cfg::TILE_BYTES + c * 16384, &p.tmap_q, h * D + c * 64, b * p.T + q0 + x * QT, q_full);
      for (int t = 0; t < n_tiles; ++t) {
        const int row = b * p.S + tile_of(t) * KT;
        const int ks = t & 1;
        if (!mbar_wait(&k_empty[ks], ((t >> 1) & 1) ^ 1, abort_flag, st, KID_ATTN_FWD, 1)) break;
        mbar_expect_tx(&k_full[ks], Cfg::TILE_BYTES);
        for (int c = 0; c < DC; ++c)
          tma_load_2d(sK + ks * Cfg::TILE_BYTES + c * 16384, &p.tmap_kv_k, g * D + c * 64, row, &k_full[ks]);
        if (!mbar_wait(&v_empty[ks], ((t >> 1) & 1) ^ 1, abort_flag, st, KID_ATTN_FWD, 2)) break;
        mbar_expect_tx(&v_full[ks], Cfg::TILE_BYTES);
        for (int c = 0; c < DC; ++c)
          tma_load_2d(sV + ks * Cfg::TILE_BYTES + c * 16384, &p.tmap_kv_v, g * D + c * 64, row, &v_full[ks]);
      }
    }
  } else if (warp == 17) {
    // -------------------------------------------------------------- MMA issuer
    if (elect_one() && n_tiles > 0) {
      const uint32_t idesc_s = make_idesc(FMT_BF16, FMT_BF16, 128, KT, false, false);
      const uint32_t idesc_pv = make_idesc(FMT_BF16, FMT_BF16, 128, D, false, true);
      bool ok = true;
      // Operand descriptors, advanced by address alone (the low word, in units of 16 bytes): what
      // this one thread does between a tile's P and its next S is time the tensor core waits.
      const uint64_t dq = make_smem_desc(smem_u32(sQ), 0, 1024, 2), dk = make_smem_desc(smem_u32(sK), 0, 1024, 2);
      const uint64_t dv = make_smem_desc(smem_u32(sV), 16384, 1024, 2);
      auto active = [&](int x, int j) { return j >= lo[x] && j < hi[x]; };
      int next_s[2] = {lo[0], lo[1]};  // next key tile whose S_x has not been issued
      int done[2] = {0, 0};            // tiles processed per query tile (for barrier parities)
      auto wait_k = [&](int j) {
        const int t = slot_of(j);
        ok = ok && mbar_wait(&k_full[t & 1], (t >> 1) & 1, abort_flag, st, KID_ATTN_FWD, 3);
      };
      // S_x(j) = Q_x · K_j^T (K_j has arrived); frees K_j when x is its last user
      auto issue_s = [&](int x, int j) {
        const int ks = slot_of(j) & 1;
        const uint64_t a0 = dq + (uint64_t)(x * (Cfg::TILE_BYTES >> 4)), b0 = dk + (uint64_t)(ks * (Cfg::TILE_BYTES >> 4));
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
          const uint32_t off = ((kk >> 2) * 16384 + (kk & 3) * 32) >> 4;
          mma_f16(tmem_base + x * 128, a0 + off, b0 + off, idesc_s, kk > 0);
        }
        tc_commit(&s_full[x]);
        next_s[x] = j + 1;
        // K_j is free once every query tile that uses it has issued its S_x(j)
        const int other = x ^ 1;
        if (!active(other, j) || next_s[other] > j) tc_commit(&k_empty[ks]);
      };
      ok = mbar_wait(q_full, 0, abort_flag, st, KID_ATTN_FWD, 4);
      // a query tile's first S is issued when the walk reaches its first key tile (at once for
      // the tile that starts the walk): issuing it earlier would wait for a key tile that the
      // two-stage ring cannot hold yet
      wait_k(j_lo);
      tc_fence_after();
#pragma unroll
      for (int x = 0; x < 2; ++x)
        if (ok && hi[x] > lo[x] && lo[x] == j_lo) issue_s(x, j_lo);
      for (int j = j_lo; j < j_hi && ok; ++j) {
        if (j >= gap_at && j < gap_at + gap) continue;
        const int t = slot_of(j), vs = t & 1;
#pragma unroll
        for (int x = 0; x < 2; ++x)
          if (ok && hi[x] > lo[x] && lo[x] == j && next_s[x] == j && j != j_lo) {
            wait_k(j);
            tc_fence_after();
            if (ok) issue_s(x, j);
          }
        ok = ok && mbar_wait(&v_full[vs], (t >> 1) & 1, abort_flag, st, KID_ATTN_FWD, 6);
        const uint64_t b0 = dv + (uint64_t)(vs * (Cfg::TILE_BYTES >> 4));
#pragma unroll
        for (int x = 0; x < 2; ++x) {
          if (!ok || !active(x, j)) continue;
          const bool more = j + 1 < hi[x];
          if (more) wait_k(j + 1);   // before P is waited for: nothing but the MMAs is left to do after it
#pragma unroll
          for (int part = 0; part < 2; ++part) {
            ok = ok && mbar_wait(&p_ready[x * 2 + part], done[x] & 1, abort_flag, st, KID_ATTN_FWD, 5);
            if (!ok) break;
            tc_fence_after();
#pragma unroll
            for (int i = 0; i < KT / 32; ++i) {
              // keys 0-31 and 64-95, then 32-63 and 96-127. P of keys 0-63 lies in the first 32 of S's
              // columns, that of keys 64-127 in columns 64-95
              const int kk = (i >> 1) * 4 + part * 2 + (i & 1);
              const uint32_t a_tmem = tmem_base + x * 128 + (kk >> 2) * 64 + (kk & 3) * 8;
              mma_f16_ts(tmem_base + 256 + x * 128, a_tmem, b0 + (uint64_t)(kk * (2048 >> 4)), idesc_pv,
                         (done[x] > 0 || part > 0 || i > 0) ? 1u : 0u);
            }
          }
          if (!ok) continue;
          ++done[x];
          if (more) issue_s(x, j + 1);
          else tc_commit(&pv_full[x]);
          if (x == 1 || !active(1, j)) tc_commit(&v_empty[vs]);
        }
      }
    }
  } else if (warp < FWD_SOFTMAX_WARPS) {
    reg_inc<FWD_SOFTMAX_REGS>();
    // -------------------------------------------------------------- softmax warps
    const int x = warp >> 3, half = (warp >> 2) & 1, quad = warp & 3, lane = threadIdx.x & 31;
    const int r = quad * 32 + lane;          // row of the tile = TMEM lane
    const int q = q0 + x * QT + r;
    const int pair = 1 + x * 4 + quad;       // named barrier of the two warps that share these rows
    const uint32_t lane_addr = (uint32_t)(quad * 32) << 16;
    const uint32_t t_s = tmem_base + x * 128 + half * 64 + lane_addr;
    const uint32_t t_o = tmem_base + 256 + x * 128 + half * (D / 2) + lane_addr;
    const int mine = (x * 2 + half) * 128 + r;   // this thread's entry; the other half's is mine ^ 128
    // with a negative scale the scores change sign first: the largest product is then the largest score
    const float sc = fabsf(p.scale_log2);
    const uint32_t flip = p.scale_log2 < 0.f ? 0x80000000u : 0u;
    float m_ref = -INFINITY, l = 0.f;
    bool ok = true;
    const int hi_key = min(p.causal ? q + shift : p.S - 1, p.S - 1) - half * 64;   // in this half's columns
    int lo_key = p.window > 0 ? q + shift - p.window + 1 : 0;
    if (p.row_lo != nullptr && q < p.T) lo_key = max(lo_key, p.row_lo[(size_t)b * p.T + q]);
    lo_key -= half * 64;
    int done = 0;
    for (int j = lo[x]; j < hi[x]; ++j, ++done) {
      const int kv0 = j * KT;
      ok = warp_all(mbar_wait(&s_full[x], done & 1, abort_flag, st, KID_ATTN_FWD, 7));
      const bool masked = flip != 0 || !warp_all(kv0 + 63 <= hi_key && kv0 >= lo_key);   // some key of the half is hidden from some row
      // S_j complete implies P·V of tile j-1 complete (same issue queue): O may be touched
      tc_fence_after();
      const int lo_c = lo_key - kv0, hi_c = hi_key - kv0;   // visible columns of this half: [lo_c, hi_c]
      auto score = [&](auto checked, uint32_t raw, int c) {
        if (!decltype(checked)::value) return __uint_as_float(raw);
        return c > hi_c || c < lo_c ? -INFINITY : __uint_as_float(raw ^ flip);
      };
      float mx = -INFINITY;
      uint32_t v[32];
      auto maximum = [&](auto checked) {
        uint32_t w[32];
        tmem_ld_x32(t_s, v);
        tmem_ld_x32(t_s + 32, w);
        tmem_ld_wait();
        float top[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int i = 0; i < 32; ++i) top[i & 3] = fmaxf(top[i & 3], fmaxf(score(checked, v[i], i), score(checked, w[i], 32 + i)));
        mx = fmaxf(fmaxf(top[0], top[1]), fmaxf(top[2], top[3]));
        // no number (a scale that is none, 0 · inf) counts as no maximum: P then is no number by itself
        if (mx != -INFINITY) mx = fmaxf(mx * sc, -INFINITY);
      };
      if (ok) {
        // two bodies: the checks would cost the tiles that need none two instructions per score
        if (masked) maximum(Flag<true>()); else maximum(Flag<false>());
      }
      // Both halves of a row see the same maximum, so they move its reference together. A warp whose
      // wait ran out says so with a NaN (a maximum never is one): the two leave the loop together.
      const int buf = (done & 1) * 512;
      row_max[buf + mine] = ok ? mx : __int_as_float(0x7fffffff);
      pair_sync(pair);
      const float theirs = row_max[buf + (mine ^ 128)];
      if (!ok || theirs != theirs) { ok = false; break; }
      const float m_row = fmaxf(mx, theirs);
      const bool move = m_row > m_ref + RESCALE_THRESHOLD;   // the first visible key always moves it
      if (__any_sync(0xffffffffu, move)) {
        const float alpha = move ? (m_ref == -INFINITY ? 0.f : exp2f(m_ref - m_row)) : 1.f;
        if (done > 0) {
#pragma unroll 1
          for (int c = 0; c < D / 2; c += 16) {
            uint32_t w[16];
            tmem_ld_x16(t_o + c, w);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 16; ++i) w[i] = __float_as_uint(__uint_as_float(w[i]) * alpha);
            tmem_st_x16(t_o + c, w);
          }
          tmem_st_wait();
        }
        l *= alpha;
        if (move) m_ref = m_row;
      }
      // P in two parts of 32 keys: the tensor core takes the first while the second is worked on
      const float nref = m_ref == -INFINITY ? 0.f : -m_ref;
      const float2 sc2 = make_float2(sc, sc), nref2 = make_float2(nref, nref);
      float2 sum0 = make_float2(0.f, 0.f), sum1 = make_float2(0.f, 0.f);
      auto probabilities = [&](auto checked, int part) {
        uint32_t packed[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const float2 s2 = make_float2(score(checked, v[2 * i], part * 32 + 2 * i), score(checked, v[2 * i + 1], part * 32 + 2 * i + 1));
          const float2 e = fma2(s2, sc2, nref2);
          float2 pr = make_float2(ex2_approx(e.x), ex2_approx(e.y));
          if (decltype(checked)::value) {   // whatever the scale (0 · -inf is no number)
            if (s2.x == -INFINITY) pr.x = 0.f;
            if (s2.y == -INFINITY) pr.y = 0.f;
          }
          if (i & 1) sum1 = add2(sum1, pr); else sum0 = add2(sum0, pr);
          packed[i] = pack_bf16(pr.x, pr.y);
        }
        tmem_st_x16(t_s + part * 16, packed);
      };
#pragma unroll
      for (int part = 0; part < 2; ++part) {
        if (part == 1) tmem_ld_x32(t_s + 32, v);   // again: held since the maximum, they would not fit the registers
        if (part == 1) tmem_ld_wait();
        if (masked) probabilities(Flag<true>(), part); else probabilities(Flag<false>(), part);
        tmem_st_wait();
        tc_fence_before();
        mbar_arrive(&p_ready[x * 2 + part]);
      }
      sum0 = add2(sum0, sum1);
      l += sum0.x + sum0.y;
    }
    if (ok && done > 0) ok = warp_all(mbar_wait(&pv_full[x], 0, abort_flag, st, KID_ATTN_FWD, 8));
    row_sum[mine] = l;
    pair_sync(pair);
    l += row_sum[mine ^ 128];
    float m_tot = m_ref, scale_o = 1.f;
    if (p.sinks) {
      const float sk = p.sinks[h] * LOG2E;
      m_tot = fmaxf(m_ref, sk);
      const float keep = m_ref == -INFINITY ? 0.f : exp2f(m_ref - m_tot);
      l = l * keep + exp2f(sk - m_tot);
      scale_o = keep;
    }
    const float inv = l > 0.f ? scale_o / l : 0.f;
    // O as bf16 into the Q tile, in TMA's swizzled layout: the tile's last P·V is complete, so Q has been
    // read. A warp's 32 rows x 64 columns are one 4 KB slab; with heads of 64 the two halves fill one
    // together. A tile without keys has waited for nothing: its Q may still be on its way into that
    // memory (the other tile's keys make the producer load both), so its zeros leave from registers.
    const bool by_tma = done > 0 && q0 + x * QT + QT <= p.T;   // and the tile ends inside the row of tokens
    uint8_t* slab = sQ + x * Cfg::TILE_BYTES + (D == 128 ? half * 16384 : 0) + quad * 4096 + lane * 128;
    __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(p.o) + (((size_t)b * p.T + (q < p.T ? q : 0)) * p.H + h) * D + half * (D / 2);
    if (ok) {
      if (done > 0) tc_fence_after();
#pragma unroll
      for (int c = 0; c < D / 2; c += 32) {
        uint32_t w[32];
        if (done > 0) {
          tmem_ld_x32(t_o + c, w);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) w[i] = 0u;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          uint4 o4;
          o4.x = pack_bf16(__uint_as_float(w[8 * k]) * inv, __uint_as_float(w[8 * k + 1]) * inv);
          o4.y = pack_bf16(__uint_as_float(w[8 * k + 2]) * inv, __uint_as_float(w[8 * k + 3]) * inv);
          o4.z = pack_bf16(__uint_as_float(w[8 * k + 4]) * inv, __uint_as_float(w[8 * k + 5]) * inv);
          o4.w = pack_bf16(__uint_as_float(w[8 * k + 6]) * inv, __uint_as_float(w[8 * k + 7]) * inv);
          const int sl = (D == 128 ? 0 : half * 4) + c / 8 + k;
          if (by_tma) *reinterpret_cast<uint4*>(slab + ((sl ^ (lane & 7)) << 4)) = o4;
          else if (q < p.T) *reinterpret_cast<uint4*>(dst + c + 8 * k) = o4;
        }
      }
    }
    if (by_tma) {
      fence_proxy_async_smem();
      if (D == 128) __syncwarp(); else pair_sync(pair);
      if (ok && lane == 0 && (D == 128 || half == 0)) {
        tma_store_2d(&p.tmap_o, slab, h * D + (D == 128 ? half * 64 : 0), b * p.T + q0 + x * QT + quad * 32);
        tma_store_commit();
        tma_store_wait_all();
      }
    }
    if (ok && half == 0 && q < p.T)
      p.lse[((size_t)b * p.H + h) * p.T + q] = l > 0.f ? (m_tot + log2f(l)) * LN2 : -INFINITY;
  }

  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    for (int i = 0; i < 64; ++i) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == 17) { tc_fence_after(); tmem_dealloc(tmem_base, Cfg::TMEM_COLS); }
}

template <int D>
static const char* attn_fwd_launch_d(const AttnArgs& a, cudaStream_t stream) {
  using Cfg = AttnFwdCfg<D>;
  AttnFwdParams p;
  const char* err;
  if ((err = make_tmap_2d(&p.tmap_q, a.q, 2, (uint64_t)a.B * a.T, (uint64_t)a.H * D, (uint64_t)a.H * D * 2, 64, QT))) return err;
  if ((err = make_tmap_2d(&p.tmap_kv_k, a.k, 2, (uint64_t)a.B * a.S, (uint64_t)a.G * D, (uint64_t)a.G * D * 2, 64, KT))) return err;
  if ((err = make_tmap_2d(&p.tmap_kv_v, a.v, 2, (uint64_t)a.B * a.S, (uint64_t)a.G * D, (uint64_t)a.G * D * 2, 64, KT))) return err;
  if ((err = make_tmap_2d(&p.tmap_o, a.o, 2, (uint64_t)a.B * a.T, (uint64_t)a.H * D, (uint64_t)a.H * D * 2, 64, 32))) return err;
  p.o = a.o; p.lse = a.lse; p.sinks = a.sinks; p.status = a.status;
  p.row_lo = a.row_lo;
  p.B = a.B; p.T = a.T; p.S = a.S; p.H = a.H; p.G = a.G;
  p.scale_log2 = a.scale * LOG2E; p.causal = a.causal ? 1 : 0; p.window = a.window; p.by_length = attn_by_length(a);
  auto kern = attn_fwd_kernel<D>;
  static bool configured[64] = {};
  if (!allow_dynamic_smem(kern, Cfg::SMEM_BYTES, configured))
    return "cudaFuncSetAttribute(max dynamic shared memory) failed";
  // the register split counts on what the compiler gave the block; with less its increase would wait for ever
  static const bool enough = [&] {
    cudaFuncAttributes attr;
    return cudaFuncGetAttributes(&attr, kern) == cudaSuccess && attr.numRegs >= FWD_LAUNCH_REGS;
  }();
  if (!enough) return "the attention kernel was compiled with fewer registers than its split hands out";
  const long grid = (long)((a.T + 2 * QT - 1) / (2 * QT)) * a.H * a.B;
  if (grid >= (1L << 31)) return "too many query tiles for one launch";
  kern<<<(unsigned)grid, FWD_THREADS, Cfg::SMEM_BYTES, stream>>>(p);
  return cudaGetLastError() == cudaSuccess ? nullptr : "attention forward launch failed";
}

const char* attn_fwd_launch(const AttnArgs& a, cudaStream_t stream) {
  if (a.H % a.G != 0) return "query heads must be a multiple of key/value heads";
  if (a.D == 128) return attn_fwd_launch_d<128>(a, stream);
  if (a.D == 64) return attn_fwd_launch_d<64>(a, stream);
  return "head_dim must be 64 or 128";
}

}  // namespace bux
