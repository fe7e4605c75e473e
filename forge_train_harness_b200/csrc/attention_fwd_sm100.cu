// Causal GQA flash attention, forward, for sm_100a on the packed kv-group-major QKV activation.
//
// Persistent and warp-specialised.  A work item is two 128-row query tiles ("0" and "1") that read the same K / V blocks:
// two heads of a KV group at the same query rows when the group size is even, two consecutive query tiles of one head
// otherwise, a single tile when the call has too few tiles to give every SM a pair.  Roles of the 20 warps:
//   warps 0-15   softmax and epilogue, two warpgroups per tile; a thread owns one query row and 64 keys at a time;
//   warp 16      TMA producer (Q tiles; K and V tiles through a ring each);
//   warps 17, 18 MMA issuers of tile 0 / tile 1 (17 owns the tensor memory); warp 19 idle (registers are re-split per four warps).
// S = Q K^T is a tcgen05.mma into tensor memory; the softmax warps read it with tcgen05.ld, run the online softmax in the log2
// domain and write P as packed bf16 over it, and O += P V takes its A operand from there.  O is rescaled in place only when
// a row's running maximum moved by more than 2^8 (the stale maximum keeps P bounded by 256).
// Returns the log-sum-exp per row so the backward never replays the forward (the reference's forward drops it and its
// backward re-runs flash-attn under autograd: forward.py:233-235, backward.py:518-527).
//
// Two shapes of the block loop, by what fits the 512 tensor-memory columns beside O:
//   head_dim 64    64-key blocks, three S / P buffers per tile; a tile's warpgroups take the even and the odd blocks and hand the
//                  running maximum on through shared memory.  The next S is always there and P waits for nothing.
//   head_dim 128   128-key blocks, one S / P buffer per tile; the warpgroups take 64 keys each and swap their row maxima; a
//                  tile's next S is issued behind its P V, under the other tile's softmax.
//
// What bounds it: per 2 x 128 queries x 128 keys 32768 exponentials = 2048 cycles of the SM's exp2 unit (a share goes to the
// FMA pipe as a polynomial in packed fp32 pairs: kPolyPairs), 1280 (D = 64) or 2080 (D = 128) cycles of products, and the
// chain product -> tcgen05.ld -> softmax -> tcgen05.st -> product, whose hand-overs cost about 400 cycles each (8 products
// alone: 262 cycles of throughput, 658 until their barrier is seen).  Measured, cycles per such block: two warpgroups of
// whole rows 2900-3300 (a warp's exponential loop alone runs at 0.4 instructions per cycle), 128-key blocks with a separate
// P at D = 64 2900 (P waits for the previous P V), 64-key blocks with two buffers 3350 (D = 64) and 4450 (D = 128).
// The next item's loads and first products run under an item's last blocks (persistent loop, heaviest items first, snake
// order over the CTAs).
//
// Replaces flash_attn_func (FA2, mma.sync) at forward.py:204-235.  Q / K / V are read in place from the QKV GEMM output through
// one 2-D tensor map (no .contiguous() copies of K and V, forward.py:83-93).
#include <type_traits>
#include <cuda.h>
#include <cuda_runtime.h>

#include "sm100_ptx.cuh"

namespace fth {

int make_tmap_bf16_2d(CUtensorMap* out, const void* ptr, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t box_rows,
                      uint32_t box_cols);

constexpr float kRescaleThreshold = 8.0f;
constexpr int kFwdThreads = 640;
// Register split of the 96 x 640 a launch gets: four softmax warpgroups, one with the producer and the issuer.
constexpr int kFwdRegsSoftmax = 104, kFwdRegsMisc = 64;
static_assert(4 * kFwdRegsSoftmax + kFwdRegsMisc <= 5 * 96, "register split exceeds the launch's registers");

template <int D>
struct FwdSmem {
  static constexpr int kBlk = (D == 64) ? 64 : 128;     // keys of a block (of one S product)
  static constexpr int kBufs = (D == 64) ? 3 : 1;       // S / P buffers per tile
  static constexpr int kQTile = 128 * D * 2;            // one 128 x D bf16 query tile
  static constexpr int kTile = kBlk * D * 2;            // one K or V tile
  static constexpr int kRing = (D == 64) ? 3 : 2;       // K tiles and V tiles in flight, each
  static constexpr int kQOff = 0;                        // Q of tile 0, Q of tile 1
  static constexpr int kKVOff = 2 * kQTile;              // per ring slot: a V tile, a K tile
  static constexpr int kMOff = kKVOff + 2 * kRing * kTile;  // row maxima: [2 tiles][2 warpgroups][128 rows]
  static constexpr int kLOff = kMOff + 2048;             // row sums, same shape
  static constexpr int kBarOff = kLOff + 2048;
  static constexpr int kTotal = kBarOff + 512 + 1024;
};

__device__ __forceinline__ uint64_t desc64(uint32_t lo, uint32_t hi) {
  uint64_t d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "r"(lo), "r"(hi));
  return d;
}

// Which tiles a work item covers.  Items are numbered heaviest (latest query rows) first.
struct FwdPlan {
  int S, B, n_kv, g;
  int mode;    // 0: two heads of a group, 1: two consecutive query tiles, 2: one tile
  int inner;   // items per query-row position
  int n_pos;   // query-row positions
  int total;
};
struct FwdItem {
  int b, j;          // batch, kv head
  int head[2];       // query head index inside the group (kv-group-major order j * g + head)
  int q0[2];         // first query row
  int spans;         // 128-key spans both tiles run over (of two consecutive tiles the first runs one that is all masked)
};
// Consecutive tiles are paired from the last one down; with an odd number of tiles the first stands in for its own partner
// (same rows twice, stored once), so that every item of a plan has the same number of tiles.
__host__ __device__ __forceinline__ int fwd_item_spans(const FwdPlan& p, int pos) {
  return p.mode == 1 ? 2 * pos + ((p.S / 128) % 2 ? 1 : 2) : pos + 1;
}
__host__ __device__ __forceinline__ void fwd_item(const FwdPlan& p, int idx, FwdItem& it) {
  const int pos = p.n_pos - 1 - idx / p.inner;
  int r = idx % p.inner;
  it.spans = fwd_item_spans(p, pos);
  if (p.mode == 0) {
    const int hg = p.g / 2;
    const int hp = r % hg;
    r /= hg;
    it.head[0] = 2 * hp;
    it.head[1] = 2 * hp + 1;
  } else {
    it.head[0] = it.head[1] = r % p.g;
    r /= p.g;
  }
  it.q0[1] = (it.spans - 1) * 128;
  it.q0[0] = (p.mode == 1 && it.spans > 1) ? it.q0[1] - 128 : it.q0[1];
  it.j = r % p.n_kv;
  it.b = r / p.n_kv;
}
// The k-th item of CTA `c` of `n`: forward in even rounds, backward in odd ones, which evens out sorted item sizes.
__device__ __forceinline__ int fwd_item_index(int k, int c, int n) { return k * n + ((k & 1) ? n - 1 - c : c); }

// Barrier poll / wait on a shared-memory address.  An issuer is one thread next to four busy softmax warps, where an instruction
// costs it 10 to 20 cycles and a barrier poll about 100: its loop is written to need few of them (addresses are constants
// off one base register), the polls of a block go out together, and each tile has an issuer of its own.
__device__ __forceinline__ uint32_t mbar_test_at(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
               : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
  return ok;
}
__device__ __forceinline__ bool mbar_wait_at(uint32_t bar, uint32_t parity, volatile int* abort_flag, int* status, int code) {
  long long t0 = 0;
  for (uint32_t spins = 1;; ++spins) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
                 : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    if (ok) return true;
    if ((spins & 1023) == 0) {
      if (*abort_flag) return false;
      const long long now = clock64();
      if (t0 == 0) t0 = now;
      if (now - t0 > kSpinLimitCycles) {
        report_status(status, code);
        *abort_flag = 1;
        return false;
      }
    }
  }
}
__device__ __forceinline__ void umma_commit_at(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ float fmax3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&v);
}
// Packed pairs of fp32 (one instruction for two lanes' worth of FMA-pipe work).
__device__ __forceinline__ uint64_t pk2(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpk2(uint64_t v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// 2^x for a pair on the FMA pipe: x = n + f with n = round(x) (the 1.5 * 2^23 trick leaves n in the low mantissa bits) and
// f in [-1/2, 1/2]; 2^f by the degree-5 minimax polynomial in relative error (Remez exchange on [-1/2, 1/2], maximum error
// 7.5e-8, the rounding level of fp32); n is added to the exponent field.  x is clamped at -125: such a P is below any
// bf16 that matters next to the row maximum's 2^-8.
__device__ __forceinline__ void exp2_poly2(float xa, float xb, float& e0, float& e1) {
  const uint64_t x2 = pk2(fmaxf(xa, -125.f), fmaxf(xb, -125.f));
  const uint64_t t2 = add2(x2, pk2(12582912.f, 12582912.f));
  const uint64_t n2 = add2(t2, pk2(-12582912.f, -12582912.f));
  const uint64_t f2 = fma2(n2, pk2(-1.f, -1.f), x2);
  uint64_t p = pk2(0.0013276472454890609f, 0.0013276472454890609f);
  p = fma2(p, f2, pk2(0.009675540961325169f, 0.009675540961325169f));
  p = fma2(p, f2, pk2(0.05550713092088699f, 0.05550713092088699f));
  p = fma2(p, f2, pk2(0.24022120237350464f, 0.24022120237350464f));
  p = fma2(p, f2, pk2(0.6931469440460205f, 0.6931469440460205f));
  p = fma2(p, f2, pk2(1.0000001192092896f, 1.0000001192092896f));
  float ta, tb, pa, pb;
  unpk2(t2, ta, tb);
  unpk2(p, pa, pb);
  e0 = __uint_as_float((__float_as_uint(ta) << 23) + __float_as_uint(pa));
  e1 = __uint_as_float((__float_as_uint(tb) << 23) + __float_as_uint(pb));
}

// Pairs out of every 8 (16 scores) whose exponentials run on the FMA pipe instead of the exp2 unit: one at head_dim 64, where that
// unit is the bound (microbenchmark of the loop, cycles per 2 warps x 64 scores: 1040 / 933 / 915 with 0 / 1 / 2 pairs); none at
// head_dim 128, where the chain of products is.
template <int D>
struct FwdTune {
  static constexpr int kPolyPairs = (D == 64) ? 1 : 0;
};

template <int D>
__global__ void __launch_bounds__(kFwdThreads, 1)
flash_fwd_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_kv,
                 __nv_bfloat16* __restrict__ out, float* __restrict__ lse_out, const FwdPlan plan, float scale_log2,
                 int* __restrict__ status, long long* __restrict__ dbg) {
  using L = FwdSmem<D>;
  constexpr int NR = L::kRing, NB = L::kBufs;
  constexpr bool kSplit = (D == 128);   // the two warpgroups of a tile split every block (otherwise they alternate)
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::kBarOff);
  uint64_t* v_full = bars;              // [NR]
  uint64_t* v_empty = v_full + NR;      // [NR]
  uint64_t* k_full = v_empty + NR;      // [NR]
  uint64_t* k_empty = k_full + NR;      // [NR]
  uint64_t* q_full = k_empty + NR;      // [2]
  uint64_t* q_empty = q_full + 2;       // [2] the tile's last S of the item has read Q
  uint64_t* s_full = q_empty + 2;       // [2 tiles][NB] S ready
  uint64_t* p_full = s_full + 2 * NB;   // [2][NB] P written and O rescaled where needed (4 or 8 warps)
  uint64_t* o_done = p_full + 2 * NB;   // [2][2 block parities] P V of a block finished (D = 64)
  uint64_t* o_final = o_done + 4;       // [2] last P V of the item finished
  uint64_t* o_free = o_final + 2;       // [2] O has been read by the epilogue (8 warps)
  uint64_t* m_full = o_free + 2;        // [2][4 lane quarters][2 block parities] running maximum of a block published (D = 64)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(m_full + 16);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int cta = blockIdx.x, n_cta = gridDim.x;

  if (threadIdx.x == 0) {
    const int n_iss = plan.mode == 2 ? 1 : 2;   // issuers that release a ring slot
    for (int s = 0; s < NR; ++s) { mbar_init(&v_full[s], 1); mbar_init(&k_full[s], 1); mbar_init(&v_empty[s], n_iss); mbar_init(&k_empty[s], n_iss); }
    for (int t = 0; t < 2; ++t) {
      mbar_init(&q_full[t], 1); mbar_init(&q_empty[t], 1); mbar_init(&o_done[2 * t], 1); mbar_init(&o_done[2 * t + 1], 1); mbar_init(&o_final[t], 1); mbar_init(&o_free[t], 8);
    }
    for (int i = 0; i < 2 * NB; ++i) { mbar_init(&s_full[i], 1); mbar_init(&p_full[i], kSplit ? 8 : 4); }
    for (int i = 0; i < 16; ++i) mbar_init(&m_full[i], 1);
    *abort_flag = 0;
    fence_barrier_init();
    fence_proxy_async();
  }
  if (warp == 16 && lane == 0) { tma_prefetch_desc(&tmap_q); tma_prefetch_desc(&tmap_kv); }
  if (warp == 17) { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  // tensor-memory columns of tile t, from 256 t: S / P buffers, then O
  auto tm_s = [&](int t, int b) { return tmem_base + 256 * t + L::kBlk * b; };
  auto tm_o = [&](int t) { return tmem_base + 256 * t + L::kBlk * NB; };

  if (warp >= 16) {
    setmaxnreg_dec<kFwdRegsMisc>();
    if (warp == 16) {
      // ---------------- TMA producer ----------------
      // Load order = the order the issuer first needs a tile: K of the first NB blocks, then V of a block and K of the
      // block NB further on (which may belong to a later item, whose Q goes first).
      if (elect_one()) {
        bool ok = true;
        FwdItem ki, vi;
        int kk = 0, kb = 0, kn = 0, ks = 0, vk = 0, vb = 0, vn = 0, vs = 0;   // item number, block, blocks of the item, ring slot
        uint32_t kph = 1, vph = 1, qph = 0;
        auto load_tile = [&](unsigned char* dst, int col, int row, uint64_t* full, uint64_t* empty, uint32_t parity) {
          if (!mbar_wait(empty, parity, abort_flag, status, kTimeoutSmemEmpty)) { ok = false; return; }
          mbar_expect_tx(full, L::kTile);
#pragma unroll
          for (int c = 0; c < D / 64; ++c) tma_load_2d(dst + c * (L::kBlk * 128), &tmap_kv, col + c * 64, row, full);
        };
        auto load_k = [&]() {
          if (kb == kn) {   // next item
            const int idx = fwd_item_index(kk, cta, n_cta);
            if (idx >= plan.total) { kn = kb = -1; return; }
            ++kk;
            fwd_item(plan, idx, ki);
            kn = ki.spans * (128 / L::kBlk);
            kb = 0;
#pragma unroll
            for (int t = 0; t < 2; ++t) {
              if ((t == 1 && plan.mode == 2) || !ok) continue;
              if (!mbar_wait(&q_empty[t], ((qph >> t) & 1) ^ 1, abort_flag, status, kTimeoutSmemEmpty)) { ok = false; continue; }
              qph ^= 1u << t;
              mbar_expect_tx(&q_full[t], L::kQTile);
#pragma unroll
              for (int c = 0; c < D / 64; ++c)
                tma_load_2d(smem + L::kQOff + t * L::kQTile + c * 16384, &tmap_q, (ki.j * (plan.g + 2) + ki.head[t]) * D + c * 64,
                            ki.b * plan.S + ki.q0[t], &q_full[t]);
            }
          }
          if (ok) load_tile(smem + L::kKVOff + (2 * ks + 1) * L::kTile, (ki.j * (plan.g + 2) + plan.g) * D, ki.b * plan.S + kb * L::kBlk,
                            &k_full[ks], &k_empty[ks], kph);
          ++kb;
          if (++ks == NR) { ks = 0; kph ^= 1; }
        };
        for (int i = 0; i < NB && ok && kn >= 0; ++i) load_k();
        while (ok) {
          if (vb == vn) {
            const int idx = fwd_item_index(vk, cta, n_cta);
            if (idx >= plan.total) break;
            ++vk;
            fwd_item(plan, idx, vi);
            vn = vi.spans * (128 / L::kBlk);
            vb = 0;
          }
          load_tile(smem + L::kKVOff + 2 * vs * L::kTile, (vi.j * (plan.g + 2) + plan.g + 1) * D, vi.b * plan.S + vb * L::kBlk,
                    &v_full[vs], &v_empty[vs], vph);
          ++vb;
          if (++vs == NR) { vs = 0; vph ^= 1; }
          if (ok && kn >= 0) load_k();
        }
      }
      __syncwarp();
    } else if (warp == 17 || (warp == 18 && plan.mode != 2)) {
      // ---------------- MMA issuer of tile t ----------------
      if (elect_one()) {
        constexpr uint32_t idesc_s = make_idesc_bf16(128, L::kBlk, false, false);
        constexpr uint32_t idesc_o = make_idesc_bf16(128, D, false, true);
        // descriptors: a constant high word, a low word of address / 16 (+ the MN-major chunk pitch for V)
        constexpr uint32_t kHi = (1024u >> 4) | (1u << 14) | (2u << 29);
        constexpr uint32_t kChunk = L::kBlk * 128;   // bytes of a 64-column chunk of a K / V tile
        const int t = warp - 17;
        const uint32_t kv_lo = smem_u32(smem + L::kKVOff) >> 4, q_lo = smem_u32(smem + L::kQOff + t * L::kQTile) >> 4;
        const uint32_t s0 = tm_s(t, 0), o0 = tm_o(t);
        const uint32_t bar0 = smem_u32(bars), bar_t1 = bar0 + 8 * t, bar_tn = bar0 + 8 * NB * t;
        auto at = [&](const uint64_t* b) { return bar0 + (uint32_t)(b - bars) * 8; };      // folds to base + constant
        auto at1 = [&](const uint64_t* b) { return bar_t1 + (uint32_t)(b - bars) * 8; };   // barrier [t]
        auto atn = [&](const uint64_t* b) { return bar_tn + (uint32_t)(b - bars) * 8; };   // barrier [t][NB]
        // P V of the current block, then S of the block NB further on: remaining blocks of either item, next item numbers
        int pv_rem = 0, s_rem = 0, pv_k = 0, s_k = 0;
        bool pv_first = false, ok = true;
        uint32_t n_q = 0, n_free = 1;   // parity of the next q_full / o_free wait (the first o_free wait passes)
        auto next_item = [&](int& k, int& rem) {
          const int idx = fwd_item_index(k, cta, n_cta);
          if (idx >= plan.total) return false;
          ++k;
          rem = fwd_item_spans(plan, plan.n_pos - 1 - idx / plan.inner) * (128 / L::kBlk);
          return true;
        };
        // S of the next block: `sr` K ring slot, `sb` S buffer (compile-time after unrolling)
        auto issue_s = [&](int sr, int sb) {
          const uint32_t k_lo = kv_lo + (((2 * sr + 1) * L::kTile) >> 4), d = s0 + L::kBlk * sb;
#pragma unroll
          for (int kk = 0; kk < D / 16; ++kk)
            umma_bf16_ss(d, desc64(q_lo + (((kk / 4) * 16384 + (kk % 4) * 32) >> 4), kHi),
                         desc64(k_lo + (((kk / 4) * kChunk + (kk % 4) * 32) >> 4), kHi), idesc_s, kk != 0 ? 1u : 0u);
          umma_commit_at(atn(&s_full[sb]));
          umma_commit_at(at(&k_empty[sr]));
          if (--s_rem == 0) umma_commit_at(at1(q_empty));
        };
        auto s_item = [&]() {   // the S stream enters its next item: that item's Q must have landed
          if (!next_item(s_k, s_rem)) return false;
          if (!mbar_wait_at(at1(q_full), n_q, abort_flag, status, kTimeoutSmemFull)) ok = false;
          n_q ^= 1u;
          return ok;
        };
        uint32_t round = 0;   // parity of the unrolled loop's trip = of the ring slots' and buffers' current use
        auto prologue = [&](auto ph_tag) {
          constexpr int PH = decltype(ph_tag)::value;
          if (!ok || (s_rem == 0 && !s_item())) return;
          if (!mbar_wait_at(at(&k_full[PH % NR]), 0, abort_flag, status, kTimeoutSmemFull)) { ok = false; return; }
          tc_fence_after();
          issue_s(PH % NR, PH % NB);
        };
        // one block; false at the end of the work
        auto step = [&](auto ph_tag) {
          constexpr int PH = decltype(ph_tag)::value;
          constexpr int KR = (PH + NB) % NR, BUF = PH % NB;
          if (pv_rem == 0) {
            if (!next_item(pv_k, pv_rem)) return false;
            pv_first = true;
          }
          const bool has_s = s_rem > 0 || s_item();
          if (!ok) return false;
          const uint32_t p_par = NB == 1 ? (uint32_t)(PH & 1) : round;
          const uint32_t k_par = (PH + NB) / NR ? round ^ 1 : round;
          const uint32_t got_v = mbar_test_at(at(&v_full[PH]), round), got_k = mbar_test_at(at(&k_full[KR]), k_par),
                         got_p = mbar_test_at(atn(&p_full[BUF]), p_par);
          if (!got_v && !mbar_wait_at(at(&v_full[PH]), round, abort_flag, status, kTimeoutSmemFull)) { ok = false; return false; }
          if (pv_first) {   // the epilogue has read the previous item's O
            if (!mbar_wait_at(at1(o_free), n_free, abort_flag, status, kTimeoutTmemEmpty)) { ok = false; return false; }
            n_free ^= 1u;
          }
          if (!got_p && !mbar_wait_at(atn(&p_full[BUF]), p_par, abort_flag, status, kTimeoutTmemFull)) { ok = false; return false; }
          tc_fence_after();
          const uint32_t b_lo = (kv_lo + ((2 * PH * L::kTile) >> 4)) | ((kChunk >> 4) << 16), a = s0 + L::kBlk * BUF;
          const uint32_t acc0 = pv_first ? 0u : 1u;
#pragma unroll
          for (int kk = 0; kk < L::kBlk / 16; ++kk)   // P of 16 keys = 8 columns; a 64-key half's P starts at its half of S
            umma_bf16_ts(o0, a + (kk / 4) * 64 + (kk % 4) * 8, desc64(b_lo + kk * (2048 >> 4), kHi), idesc_o, kk == 0 ? acc0 : 1u);
          pv_first = false;
          umma_commit_at(at(&v_empty[PH]));   // free once the MMAs issued so far have finished
          if (!kSplit) umma_commit_at(at(o_done) + 16 * t + 8 * (pv_rem & 1));   // the number of blocks is even: block parity
          if (--pv_rem == 0) umma_commit_at(at1(o_final));
          if (has_s) {
            if (!got_k && !mbar_wait_at(at(&k_full[KR]), k_par, abort_flag, status, kTimeoutSmemFull)) { ok = false; return false; }
            issue_s(KR, BUF);   // behind P V of the block that last used this buffer
          }
          return true;
        };
        prologue(std::integral_constant<int, 0>{});
        if constexpr (NB == 3) {
          prologue(std::integral_constant<int, 1>{});
          prologue(std::integral_constant<int, 2>{});
        }
        while (true) {
          if (!step(std::integral_constant<int, 0>{})) break;
          if (!step(std::integral_constant<int, 1>{})) break;
          if constexpr (NR == 3)
            if (!step(std::integral_constant<int, 2>{})) break;
          round ^= 1;
        }
      }
      __syncwarp();
    }
  } else {
    // ---------------- softmax: warpgroup e of tile t; a thread is one query row x 64 keys (kb: 64-key units) ----------------
    setmaxnreg_inc<kFwdRegsSoftmax>();
    const int t = warp / 8, e = (warp / 4) % 2, qw = warp % 4;
    const int r = qw * 32 + lane;
    const uint32_t lane_off = (uint32_t)(qw * 32) << 16;
    const int pair_bar = 1 + t * 4 + qw;   // named barrier of the two warps that share these rows
    float* m_slot = reinterpret_cast<float*>(smem + L::kMOff) + t * 256 + r;   // + 128 * warpgroup
    float* l_slot = reinterpret_cast<float*>(smem + L::kLOff) + t * 256 + r;
    uint64_t* m_bar = m_full + (t * 4 + qw) * 2;
    const uint32_t my_o = tm_o(t) + lane_off;
    uint32_t n_m = 0, n_pv = 0, n_item = 0;   // peer maxima waited for; P V products and number of finished items of the tile
    int buf = kSplit ? 0 : e;                 // S buffer of this warpgroup's next block
    uint32_t ph = 0;                          // and the parity of its barrier
    bool ok = true;
    const bool rec = dbg != nullptr && cta == 0 && qw == 0 && e == 0 && lane == 0;
    long long* drow = dbg + t * 8 * 64;
    FwdItem it;
    for (int k = 0; ok; ++k) {
      const int idx = fwd_item_index(k, cta, n_cta);
      if (idx >= plan.total) break;
      fwd_item(plan, idx, it);
      if (t == 1 && plan.mode == 2) break;
      const int nb = 2 * it.spans;   // 64-key units
      const int q0 = t == 0 ? it.q0[0] : it.q0[1];
      float m_own = -INFINITY, l_run = 0.f;
#define FTH_TS(i) do { if (rec && k == 0 && kb < 128) drow[(i) * 64 + kb / 2] = clock64(); } while (0)
      for (int kb = e; kb < nb; kb += 2) {   // split blocks: block kb / 2, half e
        FTH_TS(0);
        if (!mbar_wait(&s_full[t * NB + buf], ph, abort_flag, status, kTimeoutTmemFull)) { ok = false; break; }
        FTH_TS(1);
        tc_fence_after();
        const uint32_t my_s = tm_s(t, buf) + lane_off + (kSplit ? 64 * e : 0);
        uint64_t* my_p_full = &p_full[t * NB + buf];
        if constexpr (kSplit) ph ^= 1;
        else if ((buf += 2) >= NB) { buf -= NB; ph ^= 1; }
        uint32_t sr[64];
        tmem_ld_32x32(my_s, sr);
        tmem_ld_32x32(my_s + 32, sr + 32);
        tmem_wait_ld();
        FTH_TS(2);
        const int last = q0 + r - 64 * kb;   // keys after the query count as -inf
        if (64 * kb + 63 > q0) {
#pragma unroll
          for (int i = 0; i < 64; ++i)   // asm: the compiler would otherwise run the 64 selects in every block, without a branch
            asm volatile("{\n\t.reg .pred p;\n\tsetp.lt.s32 p, %1, %2;\n\t@p mov.b32 %0, 0xff800000;\n\t}" : "+r"(sr[i]) : "r"(last), "r"(i));
        }
        float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int i = 0; i < 64; i += 8) {
#pragma unroll
          for (int u = 0; u < 4; ++u) mx[u] = fmax3(mx[u], __uint_as_float(sr[i + 2 * u]), __uint_as_float(sr[i + 2 * u + 1]));
        }
        const float mb = fmaxf(fmax3(mx[0], mx[1], mx[2]), mx[3]) * scale_log2;
        float m_prev, m_use;   // the row's running maximum before this block, and the one its P is relative to
        if constexpr (kSplit) {
          m_slot[128 * e] = mb;   // the peer has read the previous block's: s_full waits for its P
          named_barrier_sync(pair_bar, 64);
          const float mx2 = fmaxf(mb, m_slot[128 * (e ^ 1)]);
          m_prev = m_own;
          m_use = (mx2 - m_prev > kRescaleThreshold) ? mx2 : m_prev;
        } else {
          m_prev = -INFINITY;
          if (kb > 0) {
            if (!mbar_wait(&m_bar[e ^ 1], n_m & 1, abort_flag, status, kTimeoutGeneric)) { ok = false; break; }
            ++n_m;
            m_prev = m_slot[128 * (e ^ 1)];
          }
          m_use = (mb - m_prev > kRescaleThreshold) ? mb : m_prev;
          m_slot[128 * e] = m_use;
          mbar_arrive_warp(&m_bar[e]);
        }
        FTH_TS(3);
        if (kb > (kSplit ? e : 0) && __any_sync(0xffffffffu, m_use != m_prev)) {
          // O holds the blocks before this one; this block's P V is not issued yet.  With alternating warpgroups P V of the
          // previous block may still run: wait for it.  A barrier per block parity, because s_full only implies that P V of
          // three blocks before is done: one barrier could be two phases behind or not, which a parity cannot tell apart.
          if constexpr (!kSplit) {
            if (!mbar_wait(&o_done[2 * t + (e ^ 1)], ((n_pv + kb - 1) >> 1) & 1, abort_flag, status, kTimeoutTmemEmpty)) { ok = false; break; }
            tc_fence_after();
          }
          const float alpha = exp2f(m_prev - m_use);
#pragma unroll 1
          for (int c = 0; c < (kSplit ? D / 32 : D / 16); ++c) {   // split blocks: each warpgroup its half of the columns
            const uint32_t col = my_o + (kSplit ? e * (D / 2) : 0) + c * 16;
            uint32_t rr[16];
            tmem_ld_32x16(col, rr);
            tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < 16; ++i) rr[i] = __float_as_uint(__uint_as_float(rr[i]) * alpha);
            tmem_st_32x16(col, rr);
          }
        }
        FTH_TS(4);
        const uint64_t sc2 = pk2(scale_log2, scale_log2), nm2 = pk2(-m_use, -m_use);
        uint64_t sum2[2] = {pk2(0.f, 0.f), pk2(0.f, 0.f)};
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          uint32_t pk[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const int q = c * 32 + 2 * i;
            float x0, x1, p0, p1;
            unpk2(fma2(pk2(__uint_as_float(sr[q]), __uint_as_float(sr[q + 1])), sc2, nm2), x0, x1);
            if ((i % 8) >= 8 - FwdTune<D>::kPolyPairs) {
              exp2_poly2(x0, x1, p0, p1);
            } else {
              p0 = exp2f(x0);
              p1 = exp2f(x1);
            }
            sum2[i % 2] = add2(sum2[i % 2], pk2(p0, p1));
            pk[i] = pack_bf16(p0, p1);
          }
          tmem_st_32x16(my_s + c * 16, pk);
        }
        float s0, s1, s2, s3;
        unpk2(sum2[0], s0, s1);
        unpk2(sum2[1], s2, s3);
        l_run = l_run * exp2f(m_own - m_use) + ((s0 + s1) + (s2 + s3));
        m_own = m_use;
        FTH_TS(5);
        tmem_wait_st();
        tc_fence_before();
        mbar_arrive_warp(my_p_full);
        FTH_TS(6);
      }
#undef FTH_TS
      if (!ok) break;
      // epilogue: the final maximum (of the last, odd, block); l over both warpgroups; O / l -> bf16, half the columns each
      float m_fin = m_own;
      if (!kSplit && e == 0) {
        if (!mbar_wait(&m_bar[1], n_m & 1, abort_flag, status, kTimeoutGeneric)) break;
        ++n_m;
        m_fin = m_slot[128];
      }
      l_run *= exp2f(m_own - m_fin);
      l_slot[128 * e] = l_run;
      named_barrier_sync(pair_bar, 64);
      const float l_tot = l_run + l_slot[128 * (e ^ 1)];
      const float inv = 1.f / l_tot;
      n_pv += nb;
      if (!mbar_wait(&o_final[t], n_item++ & 1, abort_flag, status, kTimeoutTmemFull)) break;
      tc_fence_after();
      const int head = it.j * plan.g + (t == 0 ? it.head[0] : it.head[1]);
      const int row = q0 + r;
      const bool dup = t == 1 && plan.mode == 1 && it.q0[0] == it.q0[1];
      __nv_bfloat16* dst = out + (size_t)(it.b * plan.S + row) * ((size_t)plan.n_kv * plan.g * D) + (size_t)head * D + e * (D / 2);
#pragma unroll
      for (int c = 0; c < D / 64; ++c) {
        uint32_t rr[32];
        tmem_ld_32x32(my_o + e * (D / 2) + c * 32, rr);
        tmem_wait_ld();
        if (c + 1 == D / 64) { tc_fence_before(); mbar_arrive_warp(&o_free[t]); }
        if (dup) continue;
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          float f[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) f[i] = __uint_as_float(rr[v * 8 + i]) * inv;
          store8(dst + c * 32 + v * 8, f);
        }
      }
      if (e == 0 && !dup) lse_out[((size_t)it.b * (plan.n_kv * plan.g) + head) * plan.S + row] = (m_fin + log2f(l_tot)) * 0.6931471805599453f;
    }
  }

  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    const long long t0 = clock64();
    while (clock64() - t0 < 2000000LL) { __nanosleep(200); }
    __syncthreads();
  }
  if (warp == 17) { tc_fence_after(); tmem_dealloc(tmem_base, 512); }
}

static int fwd_sm_count() {
  static int n = 0;
  if (n == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (n <= 0) n = 148;
  }
  return n;
}

// Pairs of tiles when there are enough of them for every SM (a pair hides one tile's MMAs under the other's softmax), single
// tiles otherwise: below that a tile alone on an SM finishes sooner than a pair.
static FwdPlan fwd_plan(int B, int S, int n_kv, int g, int sms) {
  FwdPlan p;
  p.S = S; p.B = B; p.n_kv = n_kv; p.g = g;
  const int n_t = S / 128;
  if ((long long)n_t * n_kv * g * B <= sms) { p.mode = 2; p.inner = B * n_kv * g; p.n_pos = n_t; }
  else if (g % 2 == 0) { p.mode = 0; p.inner = B * n_kv * (g / 2); p.n_pos = n_t; }
  else { p.mode = 1; p.inner = B * n_kv * g; p.n_pos = (n_t + 1) / 2; }
  p.total = p.inner * p.n_pos;
  return p;
}

template <int D>
static int launch_fwd(const CUtensorMap& tq, const CUtensorMap& tkv, void* out, float* lse, const FwdPlan& p, int sms, int* status, long long* dbg, cudaStream_t stream) {
  static bool set = false;
  if (!set) {
    if (cudaFuncSetAttribute(flash_fwd_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, FwdSmem<D>::kTotal) != cudaSuccess) return -20;
    set = true;
  }
  const int grid = p.total < sms ? p.total : sms;
  flash_fwd_kernel<D><<<grid, kFwdThreads, FwdSmem<D>::kTotal, stream>>>(tq, tkv, (__nv_bfloat16*)out, lse, p,
                                                                       1.4426950408889634f / sqrtf((float)D), status, dbg);
  return cudaGetLastError() == cudaSuccess ? 0 : -21;
}

}  // namespace fth

using namespace fth;

extern "C" {

static long long* g_fwd_dbg = nullptr;
// Optional timeline buffer (2 x 8 x 64 clock64 stamps of CTA 0's first item, per query tile); nullptr disables.
void fth_flash_fwd_set_debug(long long* buf) { g_fwd_dbg = buf; }

// qkv: [B*S, n_kv*(g+2)*d] bf16 packed; out: [B*S, n_kv*g*d] bf16; lse: [B, n_kv*g, S] fp32.  S % 128 == 0, d in {64,128}.
int fth_flash_fwd(const void* qkv, void* out, float* lse, int B, int S, int n_kv, int g, int d, int* status,
                  cudaStream_t stream) {
  if (S % 128 || (d != 64 && d != 128)) return -2;
  CUtensorMap tq, tkv;
  const uint64_t rs = (uint64_t)n_kv * (g + 2) * d;
  int r = make_tmap_bf16_2d(&tq, qkv, (uint64_t)B * S, rs, rs, 128, 64);
  if (r) return r;
  r = make_tmap_bf16_2d(&tkv, qkv, (uint64_t)B * S, rs, rs, d == 64 ? FwdSmem<64>::kBlk : FwdSmem<128>::kBlk, 64);
  if (r) return r;
  const int sms = fwd_sm_count();
  const FwdPlan p = fwd_plan(B, S, n_kv, g, sms);
  if (p.total <= 0) return 0;
  return d == 64 ? launch_fwd<64>(tq, tkv, out, lse, p, sms, status, g_fwd_dbg, stream)
                 : launch_fwd<128>(tq, tkv, out, lse, p, sms, status, g_fwd_dbg, stream);
}

}  // extern "C"
