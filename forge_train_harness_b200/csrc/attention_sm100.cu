// Causal GQA flash attention, backward, for sm_100a on the packed kv-group-major QKV activation (forward:
// attention_fwd_sm100.cu).  Replaces _flash_attn_backward (FA2, mma.sync) at backward.py:473-527.  Q / K / V are read in place
// from the QKV GEMM output through 2-D tensor maps, and dQ / dK / dV go straight into the packed layout the QKV wgrad / dgrad
// consume.
#include <type_traits>
#include <cuda.h>
#include <cuda_runtime.h>

#include "sm100_ptx.cuh"

namespace fth {

int make_tmap_bf16_2d(CUtensorMap* out, const void* ptr, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t box_rows,
                      uint32_t box_cols);

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  // one conversion instruction; doing the rounding with an integer add and a byte permute instead measured slower
  // (forward exp phase 1914 -> 2450 cycles per block): the integer pipe is half rate and the phase is issue bound
  __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&v);
}

// =====================================================================================================================
// Backward.
//
// Pre-pass (flash_bwd_prep_kernel): delta[b,h,s] = sum_d dO*O and lse2 = lse*log2(e), one warp per (row, head).
// Main kernel: one CTA per (batch, 128-key block n, one to four query heads of a KV group).  K and V tiles stay resident; the CTA
// walks the query blocks m >= n of its heads.  Per step, with every product on tcgen05 and every accumulator in tensor memory:
//     S^T  = K Q^T          (128 keys x 128 queries)            SS-MMA
//     dP^T = V dO^T                                              SS-MMA
//     P^T  = exp2(S^T*c - lse2[q]),  dS^T = P^T (dP^T - delta[q]) * scale      (one thread per key row)
//     dV  += P^T dO          A = P^T from tensor memory          TS-MMA   (dO tile reused as an MN-major B operand)
//     dK  += dS^T Q          A = dS^T from tensor memory         TS-MMA   (Q tile reused as an MN-major B operand)
//     dQ   = dS K            A = dS^T from shared memory as an MN-major operand, B = K tile MN-major
// Working on the transposed score tile means no operand ever needs a transposing copy: thread r owns key row r of
// S^T / dP^T, so P^T and dS^T are produced directly in the lane layout tcgen05 wants for an A operand.  dQ tiles are
// summed across the key blocks by TMA reduce-add into an fp32 image of the packed dQKV activation; dK / dV (summed over
// the query heads of a KV group, i.e. over CTAs) use the same path.  A finalize kernel rounds that image to bf16.
// =====================================================================================================================

constexpr int kBwd64Threads = 448;   // warps 0-7 compute, 8-11 drain, 12 TMA, 13 MMA
constexpr int kBwd128Threads = 768;  // 0-15 compute, 16-19 drain, 20 TMA, 21 and 22 MMA, 23 idle (registers are re-split per four warps)

__global__ void flash_bwd_prep_kernel(const __nv_bfloat16* __restrict__ o, const __nv_bfloat16* __restrict__ d_o,
                                      const float* __restrict__ lse, float* __restrict__ delta, float* __restrict__ lse2,
                                      int B, int S, int nq, int d, float scale) {
  // d / 8 lanes per (row, head): each lane one 16-byte vector of O and of dO, so a warp covers 4 items at head_dim 64.
  // Items run row-fastest inside a head, which makes the delta / lse2 writes and the lse reads contiguous.
  const int lpi = d / 8, ipw = 32 / lpi;
  const int lane = threadIdx.x % 32, sub = lane / lpi, l = lane % lpi;
  const long long rows = (long long)B * S, total = rows * nq;
  const long long warps = (long long)gridDim.x * (blockDim.x / 32);
  for (long long w0 = ((long long)blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32) * ipw; w0 < total; w0 += warps * ipw) {
    const long long w = w0 + sub;
    const bool ok = w < total;
    const int h = ok ? (int)(w / rows) : 0;
    const long long row = ok ? w % rows : 0;  // b*S + s
    float acc = 0.f;
    if (ok) {
      const size_t base = ((size_t)row * nq + h) * d + l * 8;
      float a[8], b8[8];
      load8(o + base, a);
      load8(d_o + base, b8);
#pragma unroll
      for (int e = 0; e < 8; ++e) acc += a[e] * b8[e];
    }
    for (int off = lpi / 2; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
    if (ok && l == 0) {
      const int b = (int)(row / S), sq = (int)(row % S);
      const size_t idx = ((size_t)b * nq + h) * S + sq;
      delta[idx] = acc * scale;   // pre-scaled: dS = P * (dP*scale - delta*scale) is one FFMA + one FMUL
      lse2[idx] = lse[idx] * 1.4426950408889634f;
    }
  }
}

// ---------------------------------------------------------------------------------------------------------------------
// head_dim 64 backward, software-pipelined.  The 128-query block of a step is handled as two 64-query halves with their own barriers, so the long serial chain of a step (commit -> tensor-memory
// load -> exp / dS math -> tensor-memory store -> fence -> barrier -> next MMA) of one half runs while the tensor core
// works on the other half and on the next step:
//     MMA order:  ... | dV_A dK_A (i) | S_A dP_A (i+1) | dV_B dK_B (i) | dQ (i) | S_B dP_B (i+1) | dV_A dK_A (i+1) | ...
// Warpgroup h computes half h.  dS^T lives in a double-buffered shared-memory operand and dQ in a double-buffered
// tensor-memory tile; tensor memory (512 columns): S^T 128, dP^T 128, dK 64, dV 64, dQ 64, K 32, V 32.
// ---------------------------------------------------------------------------------------------------------------------
struct Bwd64Smem {
  static constexpr int kTile = 128 * 64 * 2;
  static constexpr int kKOff = 0;
  static constexpr int kVOff = kTile;
  static constexpr int kQdOOff = 2 * kTile;              // 2 stages x (Q tile, dO tile)
  static constexpr int kDsOff = kQdOOff + 4 * kTile;     // 2 buffers x 2 chunks x [128 x 128 B]
  static constexpr int kStgOff = kDsOff + 65536;         // one [128 x 128 B] fp32 staging buffer per warpgroup
  // "augmentation" operands (see the kernel): a constant [128 x 16] tile of ones and, per stage, four [64 x 16] tiles
  // (S^T half 0 / 1, dP^T half 0 / 1) holding -lse2 / scale_log2 resp. -delta split into two bf16, all K-major, no swizzle
  static constexpr int kOnesOff = kStgOff + 32768;       // 4 KB
  static constexpr int kAugOff = kOnesOff + 4096;        // 2 stages x 4 x 2 KB
  static constexpr int kBarOff = kAugOff + 16384;
  static constexpr int kTotal = kBarOff + 512 + 1024;
};

__global__ void __launch_bounds__(kBwd64Threads, 1)
flash_bwd64_kernel(const __grid_constant__ CUtensorMap tmap_qkv, const __grid_constant__ CUtensorMap tmap_q64,
                   const __grid_constant__ CUtensorMap tmap_do64,
                   const __grid_constant__ CUtensorMap tmap_dqkv, const float* __restrict__ lse2, const float* __restrict__ delta,
                   int S, int n_kv, int g, int heads_per_cta, float scale, float scale_log2, int* __restrict__ status,
                   long long* __restrict__ dbg) {
  using L = Bwd64Smem;
  constexpr int D = 64;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::kBarOff);
  uint64_t* kv_full = bars;             // [1]
  uint64_t* q_full = bars + 1;          // [2 stages][2 query halves]: rows 64h .. 64h+63 of the Q and dO tiles
  uint64_t* q_empty = q_full + 4;       // [2][2]
  uint64_t* sdp_full = q_empty + 4;     // [2] per half: S^T and dP^T ready
  uint64_t* pds_full = sdp_full + 2;    // [2] per half: P^T, dS^T written (4 arrivals, one per warp)
  uint64_t* dq_full = pds_full + 2;     // [2] per dQ buffer
  uint64_t* dq_drained = dq_full + 2;   // [2] per dQ buffer (4 arrivals)
  uint64_t* kv_tmem = dq_drained + 1;   // K and V copied into tensor memory (4 arrivals); dq_full / dq_drained use slot 0 only
  uint64_t* aug_full = dq_drained + 2;  // [2] per stage: augmentation tiles written (4 arrivals, one per drain warp)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(aug_full + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int n_blk = S / 128;
  const int nq = n_kv * g;
  // key block 0 has the most query blocks: the longest CTAs of a sequence start first, its one-step CTAs fill the tail
  const int units = nq / heads_per_cta;
  const int n = (int)blockIdx.x / units, head0 = (int)blockIdx.x % units * heads_per_cta, b = blockIdx.y;
  const int j = head0 / g;                      // heads_per_cta divides g: one KV head per CTA
  const int q_col0 = (j * (g + 2) + head0 % g) * D, k_col = (j * (g + 2) + g) * D, v_col = k_col + D;
  const int grow0 = b * S;
  const int steps_h = n_blk - n;                // query blocks n .. n_blk-1 of a head
  const int steps = steps_h * heads_per_cta;    // the heads one after the other

  if (threadIdx.x == 0) {
    mbar_init(kv_full, 1);
    mbar_init(kv_tmem, 4);
    for (int s = 0; s < 2; ++s) {
      mbar_init(&q_full[2 * s], 1); mbar_init(&q_full[2 * s + 1], 1);
      mbar_init(&q_empty[2 * s], 1); mbar_init(&q_empty[2 * s + 1], 1);
      mbar_init(&sdp_full[s], 1); mbar_init(&pds_full[s], 4);     // one arrival per warp
      mbar_init(&dq_full[s], 1); mbar_init(&dq_drained[s], 4);
      mbar_init(&aug_full[s], 4);
    }
    *abort_flag = 0;
    fence_barrier_init();
    fence_proxy_async();
  }
  if (warp == 13) { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tm_s = tmem_base, tm_dp = tmem_base + 128, tm_dk = tmem_base + 256, tm_dv = tmem_base + 320;
  const uint32_t tm_dq0 = tmem_base + 384;  // one 64-column buffer
  // K and V as bf16 A operands in tensor memory (32 columns each): S^T = K Q^T and dP^T = V dO^T then fetch only their
  // 2 KB B operand from shared memory per MMA instead of 6 KB, and the shared-memory ports are what these MMAs wait for
  const uint32_t tm_k = tmem_base + 448, tm_v = tmem_base + 480;

  if (warp == 12) {
    if (elect_one()) {
      tma_prefetch_desc(&tmap_qkv);
      tma_prefetch_desc(&tmap_q64);
      tma_prefetch_desc(&tmap_do64);
      mbar_expect_tx(kv_full, 2 * L::kTile);
      tma_load_2d(smem + L::kKOff, &tmap_qkv, k_col, grow0 + n * 128, kv_full);
      tma_load_2d(smem + L::kVOff, &tmap_qkv, v_col, grow0 + n * 128, kv_full);
      // Q and dO arrive per query half: half h of a stage is free as soon as the dV / dK products of that half have
      // read it, half a step before the whole tile would be, which keeps the loads ahead of the shortened steps
      bool live = true;
      int q_col = q_col0, do_col = head0 * D;
      for (int st = 0, m = n; st < steps && live; ++st, ++m) {
        if (m == n_blk) { m = n; q_col += D; do_col += D; }
        const int stage = st & 1;
        const uint32_t phase = (st >> 1) & 1;
        unsigned char* sq = smem + L::kQdOOff + stage * 2 * L::kTile;
        for (int h = 0; h < 2; ++h) {
          if (!mbar_wait(&q_empty[2 * stage + h], phase ^ 1, abort_flag, status, kTimeoutSmemEmpty)) { live = false; break; }
          mbar_expect_tx(&q_full[2 * stage + h], L::kTile);
          tma_load_2d(sq + h * 8192, &tmap_q64, q_col, grow0 + m * 128 + 64 * h, &q_full[2 * stage + h]);
          tma_load_2d(sq + L::kTile + h * 8192, &tmap_do64, do_col, grow0 + m * 128 + 64 * h, &q_full[2 * stage + h]);
        }
      }
    }
    __syncwarp();
  } else if (warp == 13) {
    if (elect_one()) {
      constexpr uint32_t idesc_st = make_idesc_bf16(128, 64, false, false);   // S^T / dP^T half: 128 keys x 64 queries
      constexpr uint32_t idesc_dkv = make_idesc_bf16(128, D, false, true);
      constexpr uint32_t idesc_dq = make_idesc_bf16(128, D, true, true);
      const uint32_t k_addr = smem_u32(smem + L::kKOff), v_addr = smem_u32(smem + L::kVOff);
      bool ok = mbar_wait(kv_full, 0, abort_flag, status, kTimeoutSmemFull);
      if (ok) ok = mbar_wait(kv_tmem, 0, abort_flag, status, kTimeoutTmemFull);
      // S^T_h = K Q_h^T and dP^T_h = V dO_h^T for query half h of the tile in `stage`
      auto issue_sdp = [&](int stage, int h) {
        const uint32_t q_addr = smem_u32(smem + L::kQdOOff + stage * 2 * L::kTile) + h * 8192;
        const uint32_t do_addr = q_addr + L::kTile;
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
          umma_bf16_ts(tm_s + 64 * h, tm_k + kk * 8, make_smem_desc(q_addr + kk * 32, 0, 1024), idesc_st, kk != 0);
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
          umma_bf16_ts(tm_dp + 64 * h, tm_v + kk * 8, make_smem_desc(do_addr + kk * 32, 0, 1024), idesc_st, kk != 0);
        // fifth k-step: ones x (-lse2 / scale_log2) resp. ones x (-delta), so the accumulators already hold the exponent
        // argument and dP - delta and no thread has to fetch per-query vectors
        const uint32_t aug = smem_u32(smem + L::kAugOff + stage * 8192);
        const uint64_t ones_desc = make_smem_desc_plain(smem_u32(smem + L::kOnesOff), 128, 256);
        umma_bf16_ss(tm_s + 64 * h, ones_desc, make_smem_desc_plain(aug + h * 2048, 128, 256), idesc_st, 1u);
        umma_bf16_ss(tm_dp + 64 * h, ones_desc, make_smem_desc_plain(aug + 4096 + h * 2048, 128, 256), idesc_st, 1u);
        umma_commit(&sdp_full[h]);
      };
      // dV += P_h^T dO_h ; dK += dS_h^T Q_h  (64 queries = 4 steps of 16)
      auto issue_dkv = [&](int stage, int h, bool first) {
        const uint32_t q_addr = smem_u32(smem + L::kQdOOff + stage * 2 * L::kTile);
        const uint32_t do_addr = q_addr + L::kTile;
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
          umma_bf16_ts(tm_dv, tm_s + 64 * h + kk * 8, make_smem_desc(do_addr + (4 * h + kk) * 2048, 16384, 1024), idesc_dkv,
                       !(first && kk == 0));
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
          umma_bf16_ts(tm_dk, tm_dp + 64 * h + kk * 8, make_smem_desc(q_addr + (4 * h + kk) * 2048, 16384, 1024), idesc_dkv,
                       !(first && kk == 0));
      };
      if (ok) ok = mbar_wait(&aug_full[0], 0, abort_flag, status, kTimeoutSmemFull);
      if (ok) ok = mbar_wait(&q_full[0], 0, abort_flag, status, kTimeoutSmemFull);
      if (ok) { tc_fence_after(); issue_sdp(0, 0); }
      if (ok) ok = mbar_wait(&q_full[1], 0, abort_flag, status, kTimeoutSmemFull);
      if (ok) { tc_fence_after(); issue_sdp(0, 1); }
      const bool mrec = dbg != nullptr && blockIdx.x == 0 && blockIdx.y == 0;
#define FTH_MS(i) do { if (mrec && st < 64) dbg[(16 + (i)) * 64 + st] = clock64(); } while (0)
      for (int st = 0; st < steps && ok; ++st) {
        const int stage = st & 1, nstage = stage ^ 1;
        const uint32_t ph = st & 1;
        const bool more = st + 1 < steps;
        // ---- half A
        FTH_MS(0);
        if (!mbar_wait(&pds_full[0], ph, abort_flag, status, kTimeoutTmemFull)) { ok = false; break; }
        tc_fence_after();
        FTH_MS(1);
        issue_dkv(stage, 0, st == 0);
        umma_commit(&q_empty[2 * stage]);
        if (more) {
          if (!mbar_wait(&q_full[2 * nstage], ((st + 1) >> 1) & 1, abort_flag, status, kTimeoutSmemFull)) { ok = false; break; }
          if (!mbar_wait(&aug_full[nstage], ((st + 1) >> 1) & 1, abort_flag, status, kTimeoutSmemFull)) { ok = false; break; }
          tc_fence_after();
          FTH_MS(2);
          issue_sdp(nstage, 0);
        }
        FTH_MS(3);
        // ---- half B
        if (!mbar_wait(&pds_full[1], ph, abort_flag, status, kTimeoutTmemFull)) { ok = false; break; }
        tc_fence_after();
        FTH_MS(4);
        issue_dkv(stage, 1, false);
        umma_commit(&q_empty[2 * stage + 1]);
        // the next S^T / dP^T of this half goes first: warpgroup 1 waits for it, nobody waits for dQ
        if (more) {
          if (!mbar_wait(&q_full[2 * nstage + 1], ((st + 1) >> 1) & 1, abort_flag, status, kTimeoutSmemFull)) { ok = false; break; }
          tc_fence_after();
          issue_sdp(nstage, 1);
        }
        // ---- dQ(st) = dS K into buffer st & 1 (free once dQ(st-2) was drained)
        if (st >= 1) {   // the drain warps have read dQ(st - 1) out of the (single) buffer
          if (!mbar_wait(&dq_drained[0], (st - 1) & 1, abort_flag, status, kTimeoutTmemEmpty)) { ok = false; break; }
          tc_fence_after();
        }
        FTH_MS(5);
        const uint32_t ds_addr = smem_u32(smem + L::kDsOff + (st & 1) * 32768);
#pragma unroll
        for (int kk = 0; kk < 8; ++kk)
          umma_bf16_ss(tm_dq0, make_smem_desc(ds_addr + kk * 2048, 16384, 1024),
                       make_smem_desc(k_addr + kk * 2048, 16384, 1024), idesc_dq, kk != 0);
        umma_commit(&dq_full[0]);
        FTH_MS(6);
      }
#undef FTH_MS
    }
    __syncwarp();
  } else if (warp >= 8 && warp < 12) {
    // ---------------- drain warps: dQ of every step, then dK and dV, tensor memory -> TMA reduce-add ----------------
    const int qd = warp - 8;
    const int r = qd * 32 + lane;
    const uint32_t lane_off = (uint32_t)(qd * 32) << 16;
    unsigned char* stg = smem + L::kStgOff;               // two [128 x 128 B] chunks = the 64 fp32 columns of a tile
    const bool issuer = (threadIdx.x == 256);
    auto drain64 = [&](uint32_t tm_src, int col, int row, uint64_t* release_bar) {
      if (issuer) tma_wait_group_read<0>();
      named_barrier_sync(3, 128);
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t v[32];
        tmem_ld_32x32(tm_src + lane_off + c * 32, v);
        tmem_wait_ld();
        if (c == 1 && release_bar != nullptr) { tc_fence_before(); mbar_arrive_warp(release_bar); }   // the tile may be overwritten now
        unsigned char* rowp = stg + c * 16384 + r * 128;
#pragma unroll
        for (int p8 = 0; p8 < 8; ++p8)
          *reinterpret_cast<uint4*>(rowp + ((p8 ^ (r & 7)) * 16)) = make_uint4(v[p8 * 4], v[p8 * 4 + 1], v[p8 * 4 + 2], v[p8 * 4 + 3]);
      }
      fence_proxy_async();
      named_barrier_sync(3, 128);
      if (issuer) {
        tma_reduce_add_2d(&tmap_dqkv, stg, col, row);
        tma_reduce_add_2d(&tmap_dqkv, stg + 16384, col + 32, row);
        tma_commit_group();
      }
    };
    // Augmentation tiles.  Thread t of the 128 owns query t of a step: -lse2 / scale_log2 and -delta (the pre-pass stores
    // delta * scale) as bf16 hi + lo pairs in columns 0 and 1 of its row; the constant tile has ones in those two columns.
    const float inv_scale_log2 = 1.f / scale_log2, inv_scale = 1.f / scale;
    auto write_aug = [&](int st_for) {
      const int hd = st_for / steps_h, hq = r >> 6, ql = r & 63;
      const size_t row = ((size_t)b * nq + head0 + hd) * S + (n + st_for - hd * steps_h) * 128 + r;
      const float vs = -lse2[row] * inv_scale_log2, vd = -delta[row] * inv_scale;
      const __nv_bfloat16 s_hi = __float2bfloat16(vs), d_hi = __float2bfloat16(vd);
      const __nv_bfloat16 s_lo = __float2bfloat16(vs - __bfloat162float(s_hi)), d_lo = __float2bfloat16(vd - __bfloat162float(d_hi));
      unsigned char* base = smem + L::kAugOff + (st_for & 1) * 8192 + hq * 2048 + (ql >> 3) * 256 + (ql & 7) * 16;
      *reinterpret_cast<uint32_t*>(base) = (uint32_t)__bfloat16_as_ushort(s_hi) | ((uint32_t)__bfloat16_as_ushort(s_lo) << 16);
      *reinterpret_cast<uint32_t*>(base + 4096) = (uint32_t)__bfloat16_as_ushort(d_hi) | ((uint32_t)__bfloat16_as_ushort(d_lo) << 16);
      fence_proxy_async();
      mbar_arrive_warp(&aug_full[st_for & 1]);
    };
    {
      // one-time: zero both stages' tiles (only columns 0 and 1 are ever rewritten) and build the ones tile
      uint4* z = reinterpret_cast<uint4*>(smem + L::kAugOff);
      for (int i = r; i < 16384 / 16; i += 128) z[i] = make_uint4(0u, 0u, 0u, 0u);
      unsigned char* one_row = smem + L::kOnesOff + (r >> 3) * 256 + (r & 7) * 16;
      *reinterpret_cast<uint4*>(one_row) = make_uint4(0x3F803F80u, 0u, 0u, 0u);          // bf16 1.0, 1.0, then zeros
      *reinterpret_cast<uint4*>(one_row + 128) = make_uint4(0u, 0u, 0u, 0u);
      named_barrier_sync(3, 128);   // the zero fill of other threads' rows is complete before anybody writes values
      write_aug(0);
      if (steps > 1) write_aug(1);
    }
    bool ok = mbar_wait(kv_full, 0, abort_flag, status, kTimeoutSmemFull);
    if (ok) {
      // row r of the 128B-swizzled K / V tile -> lane r, 32 columns of packed bf16 (the layout a tensor-memory A operand has)
#pragma unroll 1
      for (int which = 0; which < 2; ++which) {
        const unsigned char* rowp = smem + (which == 0 ? L::kKOff : L::kVOff) + r * 128;
        uint32_t w[32];
#pragma unroll
        for (int p8 = 0; p8 < 8; ++p8) {
          const uint4 q4 = *reinterpret_cast<const uint4*>(rowp + ((p8 ^ (r & 7)) * 16));
          w[p8 * 4] = q4.x; w[p8 * 4 + 1] = q4.y; w[p8 * 4 + 2] = q4.z; w[p8 * 4 + 3] = q4.w;
        }
        tmem_st_32x16((which == 0 ? tm_k : tm_v) + lane_off, w);
        tmem_st_32x16((which == 0 ? tm_k : tm_v) + lane_off + 16, w + 16);
      }
      tmem_wait_st();
      tc_fence_before();
      mbar_arrive_warp(kv_tmem);
    }
    int q_col = q_col0;
    for (int st = 0, m = n; st < steps && ok; ++st, ++m) {
      if (m == n_blk) { m = n; q_col += D; }
      if (!mbar_wait(&dq_full[0], st & 1, abort_flag, status, kTimeoutTmemFull)) { ok = false; break; }
      tc_fence_after();
      // dq_full(st) also covers the S^T / dP^T products of step st + 1, so the tiles of parity st + 1 can take step st + 3
      // (and, the first time round, those of parity 0 step 2): always more than a step ahead of the MMA warp's need
      if (st == 0 && steps > 2) write_aug(2);
      if (st + 3 < steps) write_aug(st + 3);
      drain64(tm_dq0, q_col, grow0 + m * 128, &dq_drained[0]);
    }
    if (ok) {   // the last dQ commit also covers the final dK / dV accumulation
      drain64(tm_dk, k_col, grow0 + n * 128, nullptr);
      drain64(tm_dv, v_col, grow0 + n * 128, nullptr);
    }
    if (issuer) tma_wait_group<0>();
  } else if (warp < 8) {
    // ---------------- compute warps: warpgroup h owns query half h of every step ----------------
    const int qd = warp % 4, h = warp / 4;
    const int r = qd * 32 + lane;
    const uint32_t lane_off = (uint32_t)(qd * 32) << 16;
    bool ok = true;
    const bool rec = dbg != nullptr && blockIdx.x == 0 && blockIdx.y == 0 && qd == 0 && lane == 0;
    long long* drow = dbg + h * 8 * 64;
#define FTH_TS(i) do { if (rec && st < 64) drow[(i) * 64 + st] = clock64(); } while (0)
    for (int st = 0, sh = 0; st < steps && ok; ++st, ++sh) {
      if (sh == steps_h) sh = 0;
      FTH_TS(0);
      FTH_TS(6);
      if (!mbar_wait(&sdp_full[h], st & 1, abort_flag, status, kTimeoutTmemFull)) { ok = false; break; }
      FTH_TS(1);
      tc_fence_after();
      const bool diag = sh == 0;
      unsigned char* ds_row = smem + L::kDsOff + (st & 1) * 32768 + h * 16384 + r * 128;
      // Four 16-column chunks with a rolling prefetch: the tensor-memory load of chunk c+1 is in flight during the math
      // of chunk c.  The bf16 P^T / dS^T of chunk c land on columns [8c, 8c+8) of the warpgroup's own range, all of
      // which chunks <= c have already read.
      auto math = [&](auto diag_tag) {
        constexpr bool kDiag = decltype(diag_tag)::value;
        uint32_t sv[2][16], dv[2][16];
        tmem_ld_32x16(tm_s + lane_off + 64 * h, sv[0]);
        tmem_ld_32x16(tm_dp + lane_off + 64 * h, dv[0]);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          tmem_wait_ld();
          if (c == 0) FTH_TS(2);
          if (c < 3) {
            tmem_ld_32x16(tm_s + lane_off + 64 * h + (c + 1) * 16, sv[(c + 1) & 1]);
            tmem_ld_32x16(tm_dp + lane_off + 64 * h + (c + 1) * 16, dv[(c + 1) & 1]);
          }
          uint32_t pk[8], dk[8];
#pragma unroll
          for (int q4 = 0; q4 < 4; ++q4) {
            float p[4], d[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              p[e] = exp2f(__uint_as_float(sv[c & 1][q4 * 4 + e]) * scale_log2);   // the accumulator already holds S - lse
              if (kDiag) { if (r > 64 * h + c * 16 + q4 * 4 + e) p[e] = 0.f; }
              d[e] = (p[e] * scale) * __uint_as_float(dv[c & 1][q4 * 4 + e]);       // ... and dP - delta
            }
            pk[q4 * 2] = pack_bf16(p[0], p[1]); pk[q4 * 2 + 1] = pack_bf16(p[2], p[3]);
            dk[q4 * 2] = pack_bf16(d[0], d[1]); dk[q4 * 2 + 1] = pack_bf16(d[2], d[3]);
          }
          tmem_st_32x8(tm_s + lane_off + 64 * h + c * 8, pk);
          tmem_st_32x8(tm_dp + lane_off + 64 * h + c * 8, dk);
#pragma unroll
          for (int p2 = 0; p2 < 2; ++p2) {
            const int piece = c * 2 + p2;
            *reinterpret_cast<uint4*>(ds_row + ((piece ^ (r & 7)) * 16)) = make_uint4(dk[p2 * 4], dk[p2 * 4 + 1], dk[p2 * 4 + 2], dk[p2 * 4 + 3]);
          }
        }
      };
      if (diag) math(std::true_type{}); else math(std::false_type{});
      FTH_TS(3);
      tmem_wait_st();
      fence_proxy_async();
      tc_fence_before();
      mbar_arrive_warp(&pds_full[h]);
      FTH_TS(4);
      FTH_TS(5);
    }
#undef FTH_TS
  }

  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    const long long t0 = clock64();
    while (clock64() - t0 < 2000000LL) { __nanosleep(200); }
    __syncthreads();
  }
  if (warp == 13) { tc_fence_after(); tmem_dealloc(tmem_base, 512); }
}

// ---------------------------------------------------------------------------------------------------------------------
// head_dim 128 backward.  Same math, on a stream of 64-query half blocks k = 0, 1, ... of the CTA's 128-key block, so that the
// tensor core never waits for the chain  S^T -> exp -> dP^T -> dS^T  of one half: it has the other half's products to run.
//     products:  ... | dP(k+1) | dV(k) dK(k) | S(k+2), dQ(k) | dP(k+2) | dV(k+1) dK(k+1) | S(k+3), dQ(k+1) | ...
// The compute warps of parity h own the halves of parity h: the exponentials of k + 1 run under the products of k - 1, its dS^T
// under those of k.  Tensor memory (512 columns): S^T of two halves 128, dP^T 64, dQ^T 64, dK 128, dV 128.  P^T and dS^T of a
// half share the columns of its S^T, so dP^T is free as soon as it has been read.
// dQ is taken transposed, [128 d x 64 queries] = K^T dS^T: a 64-row accumulator would need twice the columns, and a warp that
// owns 32 neighbouring d of a query adds its 128 bytes straight from registers into the fp32 image (red.global; a TMA
// reduce-add through shared memory measured 3 % slower).
// Bound: the tensor core, 1740 cycles a half (measured alone: 52 cycles a 128 x 64 SS product, 64 a 128 x 128 TS product), of which
// about 60 % is reached.  1 x 4096 tokens, 32/2 heads: 659 us with one 128-query block at a time and every stage of it in
// series -> 346 us = 0.60 of the measured 1668 TFLOP/s.
// ---------------------------------------------------------------------------------------------------------------------
struct Bwd128Smem {
  static constexpr int kTile = 128 * 128 * 2;             // K, V: two 64-column chunks of 16 KB
  static constexpr int kHalf = 64 * 128 * 2;              // 64 rows of Q or dO: two 64-column chunks of 8 KB
  static constexpr int kQStages = 4, kDoStages = 3;
  static constexpr int kKOff = 0;
  static constexpr int kVOff = kTile;
  static constexpr int kQOff = 2 * kTile;                 // after the last step: staging of dK (64 KB)
  static constexpr int kDoOff = kQOff + kQStages * kHalf; // after the last step: staging of dV, with the first dS^T buffer
  static constexpr int kDsOff = kDoOff + kDoStages * kHalf;  // two [128 keys x 64 queries] bf16
  // k-step operands [rows x 16] (see flash_bwd64_kernel) of which only columns 0 and 1 are not zero: the first 16 bytes of the
  // rows lie together (128 B per 8 rows), the second 16 bytes of every row are one block of zeros shared by all of them
  static constexpr int kOnesOff = kDsOff + 2 * 16384;     // [128 x 16] with ones in columns 0, 1
  static constexpr int kAugOff = kOnesOff + 2048;         // per Q stage [64 x 16] of -lse2 / scale_log2 and of -delta
  static constexpr int kZeroOff = kAugOff + kQStages * 2048;
  static constexpr int kBarOff = kZeroOff + 2048;
  static constexpr int kTotal = kBarOff + 512 + 1024;
};
static_assert(Bwd128Smem::kTotal <= 232448, "shared memory per CTA");

__device__ __forceinline__ void red_add_f32(float* p, float v) {
  asm volatile("red.global.add.f32 [%0], %1;" ::"l"(p), "f"(v) : "memory");
}

// Register split of the 80 x 768 a launch gets: four compute warpgroups keep theirs, the drain warps take what the producer and
// the issuers give up.
constexpr int kBwd128RegsDrain = 104, kBwd128RegsMisc = 56;
static_assert(4 * 80 + kBwd128RegsDrain + kBwd128RegsMisc <= 6 * 80, "more registers than the launch has");

// The SS and TS products with operand descriptors given as words (low: address and leading offset; high: constant).
__device__ __forceinline__ void umma_bf16_ss_words(uint32_t d_tmem, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo, uint32_t b_hi,
                                                   uint32_t idesc, bool accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 a, b;\n\tsetp.ne.b32 p, %6, 0;\n\tmov.b64 a, {%1, %2};\n\tmov.b64 b, {%3, %4};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %5, p;\n\t}\n"
      ::"r"(d_tmem), "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"((uint32_t)accumulate)
      : "memory");
}
__device__ __forceinline__ void umma_bf16_ts_words(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_lo, uint32_t b_hi, uint32_t idesc,
                                                   bool accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 b;\n\tsetp.ne.b32 p, %5, 0;\n\tmov.b64 b, {%2, %3};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], b, %4, p;\n\t}\n"
      ::"r"(d_tmem), "r"(a_tmem), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"((uint32_t)accumulate)
      : "memory");
}

__global__ void __launch_bounds__(kBwd128Threads, 1)
flash_bwd128_kernel(const __grid_constant__ CUtensorMap tmap_qkv, const __grid_constant__ CUtensorMap tmap_q64,
                    const __grid_constant__ CUtensorMap tmap_do64, const __grid_constant__ CUtensorMap tmap_dqkv,
                    float* __restrict__ img, const float* __restrict__ lse2, const float* __restrict__ delta, int S, int n_kv,
                    int g, int heads_per_cta, float scale, float scale_log2, int* __restrict__ status) {
  using L = Bwd128Smem;
  constexpr int D = 128;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::kBarOff);
  uint64_t* kv_full = bars;                          // [1]
  uint64_t* q_full = bars + 1;                       // [kQStages] Q and, with 4 arrivals, the augmentation rows of the half
  uint64_t* q_empty = q_full + L::kQStages;          // [kQStages]
  uint64_t* do_full = q_empty + L::kQStages;         // [kDoStages]
  uint64_t* do_empty = do_full + L::kDoStages;       // [kDoStages]
  uint64_t* s_full = do_empty + L::kDoStages;        // [2] by parity of the half
  uint64_t* dp_full = s_full + 2;                    // [2] by parity
  uint64_t* dp_read = dp_full + 2;                   // dP^T is in registers (8 arrivals)
  uint64_t* pds_full = dp_read + 1;                  // [2] P^T, dS^T written (8 arrivals)
  uint64_t* p_free = pds_full + 2;                   // [2] dV and dK of the half have read its P^T and dS^T
  uint64_t* dq_full = p_free + 2;                    // [2] by parity
  uint64_t* dq_drained = dq_full + 2;                // 4 arrivals
  uint64_t* done = dq_drained + 1;                   // every product is finished
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int n_blk = S / 128, nq = n_kv * g;
  // key block 0 has the most query blocks: the longest CTAs of a sequence start first, its one-step CTAs fill the tail
  const int units = nq / heads_per_cta;
  const int n = (int)blockIdx.x / units, head0 = (int)blockIdx.x % units * heads_per_cta, b = blockIdx.y;
  const int j = head0 / g;                           // heads_per_cta divides g: one KV head per CTA
  const int q_col0 = (j * (g + 2) + head0 % g) * D, k_col = (j * (g + 2) + g) * D, v_col = k_col + D;
  const int grow0 = b * S;
  const int steps = n_blk - n;                       // query blocks n .. n_blk-1 of a head
  const int halves = 2 * steps * heads_per_cta;      // 64-query halves, the heads one after the other
  const int row_first = n * 128;                     // sequence position of a head's first half

  if (threadIdx.x == 0) {
    mbar_init(kv_full, 1);
    for (int s = 0; s < L::kQStages; ++s) { mbar_init(&q_full[s], 5); mbar_init(&q_empty[s], 1); }
    for (int s = 0; s < L::kDoStages; ++s) { mbar_init(&do_full[s], 1); mbar_init(&do_empty[s], 1); }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&s_full[s], 1); mbar_init(&dp_full[s], 1); mbar_init(&pds_full[s], 8);
      mbar_init(&p_free[s], 1); mbar_init(&dq_full[s], 1);
    }
    mbar_init(dp_read, 8);
    mbar_init(dq_drained, 4);
    mbar_init(done, 1);
    *abort_flag = 0;
    fence_barrier_init();
    fence_proxy_async();
  }
  if (warp == 21) { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tm_s = tmem_base, tm_dp = tmem_base + 128, tm_dq = tmem_base + 192, tm_dk = tmem_base + 256,
                 tm_dv = tmem_base + 384;

  if (warp >= 20) {
    setmaxnreg_dec<kBwd128RegsMisc>();
    if (warp == 20) {
      // ---------------- TMA producer ----------------
      if (elect_one()) {
        tma_prefetch_desc(&tmap_qkv);
        tma_prefetch_desc(&tmap_q64);
        tma_prefetch_desc(&tmap_do64);
        mbar_expect_tx(kv_full, 2 * L::kTile);
        for (int c = 0; c < 2; ++c) {
          tma_load_2d(smem + L::kKOff + c * 16384, &tmap_qkv, k_col + c * 64, grow0 + n * 128, kv_full);
          tma_load_2d(smem + L::kVOff + c * 16384, &tmap_qkv, v_col + c * 64, grow0 + n * 128, kv_full);
        }
        int qs = 0, ds = 0;
        uint32_t qph = 0, dph = 0;
        int q_col = q_col0, do_col = head0 * D;
        for (int k = 0, kh = 0; k < halves; ++k, ++kh) {
          if (kh == 2 * steps) { kh = 0; q_col += D; do_col += D; }
          const int row = grow0 + row_first + 64 * kh;
          if (!mbar_wait(&q_empty[qs], qph ^ 1, abort_flag, status, kTimeoutSmemEmpty)) break;
          mbar_expect_tx(&q_full[qs], L::kHalf);
          for (int c = 0; c < 2; ++c)
            tma_load_2d(smem + L::kQOff + qs * L::kHalf + c * 8192, &tmap_q64, q_col + c * 64, row, &q_full[qs]);
          if (++qs == L::kQStages) { qs = 0; qph ^= 1; }
          if (!mbar_wait(&do_empty[ds], dph ^ 1, abort_flag, status, kTimeoutSmemEmpty)) break;
          mbar_expect_tx(&do_full[ds], L::kHalf);
          for (int c = 0; c < 2; ++c)
            tma_load_2d(smem + L::kDoOff + ds * L::kHalf + c * 8192, &tmap_do64, do_col + c * 64, row, &do_full[ds]);
          if (++ds == L::kDoStages) { ds = 0; dph ^= 1; }
        }
      }
      __syncwarp();
    } else if (warp < 23) {
      // ---------------- two MMA issuers: warp 21 S^T and dP^T, warp 22 dV, dK and dQ^T ----------------
      // An issuer needs about 28 cycles a product and 100 a barrier poll: 2000 a half for one issuer, where the products need 1740
      // by themselves.  Operand descriptors are a constant high word and a low word plus constants.
      constexpr uint32_t kHi = (1024 >> 4) | (1u << 14) | (2u << 29);          // 8-row groups 1 KB apart, 128-byte swizzle
      const uint32_t base = smem_u32(smem) >> 4;
      const uint32_t k_lo = base + (L::kKOff >> 4), v_lo = base + (L::kVOff >> 4);
      if (warp == 21 && elect_one()) {
        constexpr uint32_t idesc_st = make_idesc_bf16(128, 64, false, false);  // 128 keys x 64 queries
        constexpr uint32_t kHiAug = (128 >> 4) | (1u << 14);                   // 8-row groups 128 B apart, no swizzle
        const uint32_t ones_lo = (base + (L::kOnesOff >> 4)) | ((uint32_t)(L::kZeroOff - L::kOnesOff) << 12);
        // x^T = A B^T for 64 queries, plus the k-step  ones x (-lse2 / scale_log2)  or  ones x (-delta)
        auto issue_st = [&](uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t aug_off) {
#pragma unroll
          for (int kk = 0; kk < D / 16; ++kk)
            umma_bf16_ss_words(d_tmem, a_lo + (((kk / 4) * 16384 + (kk % 4) * 32) >> 4), kHi,
                               b_lo + (((kk / 4) * 8192 + (kk % 4) * 32) >> 4), kHi, idesc_st, kk != 0);
          const uint32_t aug_lo = (base + (aug_off >> 4)) | ((L::kZeroOff - aug_off) << 12);
          umma_bf16_ss_words(d_tmem, ones_lo, kHiAug, aug_lo, kHiAug, idesc_st, true);
        };
        auto do_s = [&](int k) -> bool {
          const int st = k % L::kQStages;
          if (!mbar_wait(&q_full[st], (k / L::kQStages) & 1, abort_flag, status, kTimeoutSmemFull)) return false;
          tc_fence_after();
          issue_st(tm_s + 64 * (k & 1), k_lo, base + ((L::kQOff + st * L::kHalf) >> 4), L::kAugOff + st * 2048);
          umma_commit(&s_full[k & 1]);
          return true;
        };
        int ds = 0;
        uint32_t dph = 0;
        auto do_dp = [&](int k) -> bool {
          if (!mbar_wait(&do_full[ds], dph, abort_flag, status, kTimeoutSmemFull)) return false;
          tc_fence_after();
          issue_st(tm_dp, v_lo, base + ((L::kDoOff + ds * L::kHalf) >> 4), L::kAugOff + (k % L::kQStages) * 2048 + 1024);
          umma_commit(&dp_full[k & 1]);
          if (++ds == L::kDoStages) { ds = 0; dph ^= 1; }
          return true;
        };
        bool ok = mbar_wait(kv_full, 0, abort_flag, status, kTimeoutSmemFull);
        ok = ok && do_s(0) && do_s(1) && do_dp(0);
        for (int k = 0; k + 1 < halves && ok; ++k) {
          if (!mbar_wait(dp_read, k & 1, abort_flag, status, kTimeoutTmemEmpty)) break;
          if (!do_dp(k + 1)) break;
          if (k + 2 < halves) {
            if (!mbar_wait(&p_free[k & 1], (k >> 1) & 1, abort_flag, status, kTimeoutTmemEmpty)) break;
            if (!do_s(k + 2)) break;
          }
        }
      }
      if (warp == 22 && elect_one()) {
        constexpr uint32_t idesc_dkv = make_idesc_bf16(128, D, false, true);   // A from tensor memory, B MN-major
        constexpr uint32_t idesc_dq = make_idesc_bf16(128, 64, true, true);    // A = K as [d x keys], B = dS^T, both MN-major
        int ds = 0;
        for (int k = 0; k < halves; ++k) {
          const int par = k & 1, qs = k % L::kQStages;
          if (!mbar_wait(&pds_full[par], (k >> 1) & 1, abort_flag, status, kTimeoutTmemFull)) break;
          tc_fence_after();
          // dV += P^T dO ; dK += dS^T Q  (64 queries = 4 steps of 16)
          const uint32_t q_lo = (base + ((L::kQOff + qs * L::kHalf) >> 4)) | ((8192 >> 4) << 16);
          const uint32_t do_lo = (base + ((L::kDoOff + ds * L::kHalf) >> 4)) | ((8192 >> 4) << 16);
#pragma unroll
          for (int kk = 0; kk < 4; ++kk)
            umma_bf16_ts_words(tm_dv, tm_s + 64 * par + (kk / 2) * 32 + (kk % 2) * 8, do_lo + ((kk * 2048) >> 4), kHi, idesc_dkv,
                               kk != 0 || k != 0);
#pragma unroll
          for (int kk = 0; kk < 4; ++kk)
            umma_bf16_ts_words(tm_dk, tm_s + 64 * par + (kk / 2) * 32 + 16 + (kk % 2) * 8, q_lo + ((kk * 2048) >> 4), kHi, idesc_dkv,
                               kk != 0 || k != 0);
          umma_commit(&p_free[par]);
          umma_commit(&q_empty[qs]);
          umma_commit(&do_empty[ds]);
          if (++ds == L::kDoStages) ds = 0;
          if (k >= 1) {
            if (!mbar_wait(dq_drained, par ^ 1, abort_flag, status, kTimeoutTmemEmpty)) break;
            tc_fence_after();
          }
          const uint32_t ds_lo = (base + ((L::kDsOff + par * 16384) >> 4)) | ((16384 >> 4) << 16);
          const uint32_t kt_lo = k_lo | ((16384 >> 4) << 16);
#pragma unroll
          for (int kk = 0; kk < 8; ++kk)
            umma_bf16_ss_words(tm_dq, kt_lo + ((kk * 2048) >> 4), kHi, ds_lo + ((kk * 2048) >> 4), kHi, idesc_dq, kk != 0);
          umma_commit(&dq_full[par]);
        }
        umma_commit(done);
      }
      __syncwarp();
    }
  } else if (warp >= 16) {
    // ---------------- drain warps: dQ^T of every half into the fp32 image; augmentation rows ----------------
    setmaxnreg_inc<kBwd128RegsDrain>();
    const int qd = warp - 16, t = qd * 32 + lane;
    const uint32_t lane_off = (uint32_t)(qd * 32) << 16;
    // thread t < 64 writes the S^T tile's row of query t, thread 64 + t the dP^T tile's: value as bf16 high + low part.
    // The pre-pass stores delta * scale.  The rows are asked for in order: a head's halves are 64 apart, the next head's S later.
    const float* aug_src = (t < 64 ? lse2 : delta) + ((size_t)b * nq + head0) * S + row_first + (t & 63);
    int aug_k = 0;
    auto next_aug = [&]() -> float {
      const float val = *aug_src;
      aug_src += 64;
      if (++aug_k == 2 * steps) { aug_k = 0; aug_src += S - 128 * steps; }
      return val;
    };
    const float aug_mul = t < 64 ? -1.f / scale_log2 : -1.f / scale;
    auto write_aug = [&](int k, float raw) {
      const float val = raw * aug_mul;
      const __nv_bfloat16 hi = __float2bfloat16(val);
      const __nv_bfloat16 lo = __float2bfloat16(val - __bfloat162float(hi));
      const int st = k % L::kQStages;
      *reinterpret_cast<uint32_t*>(smem + L::kAugOff + st * 2048 + t * 16) =
          (uint32_t)__bfloat16_as_ushort(hi) | ((uint32_t)__bfloat16_as_ushort(lo) << 16);
      fence_proxy_async();
      mbar_arrive_warp(&q_full[st]);
    };
    {
      // one-time: zero the rows (only columns 0 and 1 are ever rewritten) and the shared zero block, and build the ones tile
      uint4* z = reinterpret_cast<uint4*>(smem + L::kAugOff);
      for (int e = t; e < (L::kBarOff - L::kAugOff) / 16; e += 128) z[e] = make_uint4(0u, 0u, 0u, 0u);
      *reinterpret_cast<uint4*>(smem + L::kOnesOff + t * 16) = make_uint4(0x3F803F80u, 0u, 0u, 0u);   // bf16 1.0, 1.0, then zeros
      named_barrier_sync(5, 128);
      for (int k = 0; k < L::kQStages && k < halves; ++k) write_aug(k, next_aug());
    }
    // dq_full(k) means that S^T and dP^T of half k are done too, so the slot of half k can take half k + 4, whose S^T is two
    // halves away.  The value is fetched one half ahead.
    float vn = L::kQStages < halves ? next_aug() : 0.f;
    const size_t rs = (size_t)n_kv * (g + 2) * D;
    float* dst = img + (size_t)(grow0 + row_first) * rs + q_col0 + t;
    for (int k = 0, kh = 0; k < halves; ++k, ++kh) {
      if (kh == 2 * steps) { kh = 0; dst += D - (ptrdiff_t)(128 * steps) * (ptrdiff_t)rs; }
      if (!mbar_wait(&dq_full[k & 1], (k >> 1) & 1, abort_flag, status, kTimeoutTmemFull)) break;
      tc_fence_after();
      uint32_t v[64];
      tmem_ld_32x32(tm_dq + lane_off, v);
      tmem_ld_32x32(tm_dq + lane_off + 32, v + 32);
      tmem_wait_ld();
      tc_fence_before();
      mbar_arrive_warp(dq_drained);
      if (k + 4 < halves) write_aug(k + 4, vn);
      if (k + 5 < halves) vn = next_aug();
#pragma unroll
      for (int e = 0; e < 64; ++e) {
        red_add_f32(dst, __uint_as_float(v[e]));
        dst += rs;
      }
    }
  } else {
    // ---------------- compute warps ----------------
    // Warpgroups 2h and 2h + 1 own the halves of parity h, 32 queries each; a thread owns one key row.  (One warpgroup per half,
    // 64 queries a thread: its chain from S^T to dS^T, 2700 cycles, held the products up; 368 -> 346 us at the size above,
    // together with two heads per CTA.)
    const int qd = warp % 4, e = (warp / 4) % 2, h = warp / 8;
    const int r = qd * 32 + lane;
    const uint32_t lane_off = (uint32_t)(qd * 32) << 16;
    const uint32_t tm_sh = tm_s + 64 * h + 32 * e + lane_off, tm_dph = tm_dp + 32 * e + lane_off;
    unsigned char* ds_row = smem + L::kDsOff + h * 16384 + r * 128;
    bool ok = true;
    for (int st = 0, sh = 0; 2 * st < halves; ++st, ++sh) {
      if (sh == steps) sh = 0;
      if (!mbar_wait(&s_full[h], st & 1, abort_flag, status, kTimeoutTmemFull)) { ok = false; break; }
      tc_fence_after();
      // P^T lands on the first 16 of the warpgroup's 32 columns of S^T, dS^T on the others
      float p[32];
      {
        uint32_t sv[32], pk[16];
        tmem_ld_32x32(tm_sh, sv);
        tmem_wait_ld();
#pragma unroll
        for (int c = 0; c < 32; ++c) p[c] = exp2f(__uint_as_float(sv[c]) * scale_log2);   // the accumulator holds S - lse
        if (sh == 0) {   // the diagonal block
#pragma unroll
          for (int c = 0; c < 32; ++c)
            if (r > 64 * h + 32 * e + c) p[c] = 0.f;
        }
#pragma unroll
        for (int c = 0; c < 16; ++c) pk[c] = pack_bf16(p[2 * c], p[2 * c + 1]);
        tmem_st_32x16(tm_sh, pk);
      }
      if (!mbar_wait(&dp_full[h], st & 1, abort_flag, status, kTimeoutTmemFull)) { ok = false; break; }
      tc_fence_after();
      {
        // all of dP^T goes to registers at once: dP^T of the next half is issued as soon as it is out
        uint32_t dv[32], dk[16];
        tmem_ld_32x32(tm_dph, dv);
        tmem_wait_ld();
        tc_fence_before();
        mbar_arrive_warp(dp_read);
#pragma unroll
        for (int c = 0; c < 16; ++c) {
          const float d0 = (p[2 * c] * scale) * __uint_as_float(dv[2 * c]);                // dP - delta
          const float d1 = (p[2 * c + 1] * scale) * __uint_as_float(dv[2 * c + 1]);
          dk[c] = pack_bf16(d0, d1);
        }
        tmem_st_32x16(tm_sh + 16, dk);
        // dQ^T of the last half of this parity has read the dS^T buffer
        if (st > 0 && !mbar_wait(&dq_full[h], (st - 1) & 1, abort_flag, status, kTimeoutTmemFull)) { ok = false; break; }
#pragma unroll
        for (int p4 = 0; p4 < 4; ++p4)
          *reinterpret_cast<uint4*>(ds_row + (((4 * e + p4) ^ (r & 7)) * 16)) =
              make_uint4(dk[p4 * 4], dk[p4 * 4 + 1], dk[p4 * 4 + 2], dk[p4 * 4 + 3]);
      }
      tmem_wait_st();
      fence_proxy_async();
      tc_fence_before();
      mbar_arrive_warp(&pds_full[h]);
    }
    // warpgroups 0 and 1 hand on dK, 2 and 3 dV, 64 columns each: through the operand rings (every load has landed and been
    // used) as [128 x 32] fp32 chunks of a TMA reduce-add
    if (ok && mbar_wait(done, 0, abort_flag, status, kTimeoutTmemFull)) {
      tc_fence_after();
      unsigned char* stg = smem + (h == 0 ? L::kQOff : L::kDoOff) + e * 32768;
#pragma unroll 1
      for (int c = 0; c < 2; ++c) {
        uint32_t v[32];
        tmem_ld_32x32((h == 0 ? tm_dk : tm_dv) + lane_off + (2 * e + c) * 32, v);
        tmem_wait_ld();
        unsigned char* rowp = stg + c * 16384 + r * 128;
#pragma unroll
        for (int p8 = 0; p8 < 8; ++p8)
          *reinterpret_cast<uint4*>(rowp + ((p8 ^ (r & 7)) * 16)) = make_uint4(v[p8 * 4], v[p8 * 4 + 1], v[p8 * 4 + 2], v[p8 * 4 + 3]);
      }
      fence_proxy_async();
      named_barrier_sync(1 + warp / 4, 128);
      if (r == 0) {
        for (int c = 0; c < 2; ++c)
          tma_reduce_add_2d(&tmap_dqkv, stg + c * 16384, (h == 0 ? k_col : v_col) + (2 * e + c) * 32, grow0 + n * 128);
        tma_commit_group();
        tma_wait_group<0>();
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    const long long t0 = clock64();
    while (clock64() - t0 < 2000000LL) { __nanosleep(200); }
    __syncthreads();
  }
  if (warp == 21) { tc_fence_after(); tmem_dealloc(tmem_base, 512); }
}

// fp32 image -> bf16 packed dQKV.  With a RoPE table the inverse rotation (the RoPE backward) of the q and k head
// slots is applied on the way, so the gradient needs no separate RoPE pass.
__global__ void dqkv_finalize_kernel(const float* __restrict__ src, __nv_bfloat16* __restrict__ dst, const float* __restrict__ table,
                                     int M, int S, int n_kv, int g, int d) {
  const int half = d / 2, vph = half / 8;
  const int slots = n_kv * (g + 2);
  const size_t total = (size_t)M * slots * vph;
  const size_t row_stride = (size_t)slots * d;
  for (size_t it = blockIdx.x * (size_t)blockDim.x + threadIdx.x; it < total; it += (size_t)gridDim.x * blockDim.x) {
    const int vec = it % vph;
    const size_t t = it / vph;
    const int sl = t % slots;
    const int row = t / slots;
    const size_t off = (size_t)row * row_stride + (size_t)sl * d + vec * 8;
    float x1[8], x2[8];
    load8(src + off, x1);
    load8(src + off + half, x2);
    if (table != nullptr && (sl % (g + 2)) <= g) {
      const float* tb = table + (size_t)(row % S) * d + vec * 8;
      float c[8], sn[8];
      load8(tb, c);
      load8(tb + half, sn);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float a = x1[i], b = x2[i];
        x1[i] = a * c[i] + b * sn[i];
        x2[i] = b * c[i] - a * sn[i];
      }
    }
    store8(dst + off, x1);
    store8(dst + off + half, x2);
  }
}

// How many query heads of a KV group a backward CTA walks.  More heads share one start (K and V tiles, filling the
// pipeline) and one dK / dV hand-over, together about 2.5 steps (49 of 368 us at 1 x 4096 tokens, 32/2 heads, one head each); but a CTA of c * n_blk steps must not be long against an SM's share of
// all steps, or the last ones to finish leave the others idle.
// head_dim 64, 4 x 4096 tokens, 16/2 heads: short CTAs first and one head each 465 us, long ones first and four heads each 421 us.
static int bwd_heads_per_cta(int n_blk, int n_kv, int g, int B) {
  const double share = (double)B * n_kv * g * n_blk * (n_blk + 1) / 2 / 148;
  int best = 1;
  for (int c = 2; c <= 4 && c <= g; ++c)
    if (g % c == 0 && c * n_blk <= 0.6 * share) best = c;
  return best;
}

int make_tmap_f32_2d(CUtensorMap* out, const void* ptr, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t box_rows,
                     uint32_t box_cols);

}  // namespace fth

using namespace fth;

extern "C" {

// Scratch: `scratch_f32` holds [B*S, qkv_dim] fp32 (zeroed here) followed by delta and lse2, each [B, nq, S] fp32.
static long long* g_bwd_dbg = nullptr;
void fth_flash_bwd_set_debug(long long* buf) { g_bwd_dbg = buf; }

size_t fth_flash_bwd_scratch_bytes(int B, int S, int n_kv, int g, int d) {
  return ((size_t)B * S * n_kv * (g + 2) * d + 2 * (size_t)B * n_kv * g * S) * sizeof(float);
}

int fth_flash_bwd(const void* d_out, const void* qkv, const void* out, const float* lse, void* dqkv, void* scratch_f32,
                  const float* rope_table, int B, int S, int n_kv, int g, int d, int* status, cudaStream_t stream) {
  if (S % 128 || (d != 64 && d != 128)) return -2;
  const int nq = n_kv * g;
  const uint64_t rs = (uint64_t)n_kv * (g + 2) * d;
  const size_t n_img = (size_t)B * S * rs;
  float* img = reinterpret_cast<float*>(scratch_f32);
  float* delta = img + n_img;
  float* lse2 = delta + (size_t)B * nq * S;
  cudaMemsetAsync(img, 0, n_img * sizeof(float), stream);
  {
    long long warps = ((long long)B * S * nq + (256 / d) - 1) / (256 / d);
    int blocks = (int)((warps + 7) / 8);
    if (blocks > 148 * 16) blocks = 148 * 16;
    flash_bwd_prep_kernel<<<blocks, 256, 0, stream>>>((const __nv_bfloat16*)out, (const __nv_bfloat16*)d_out, lse, delta, lse2,
                                                     B, S, nq, d, 1.f / sqrtf((float)d));
  }
  CUtensorMap tq, tdq;
  int r = make_tmap_bf16_2d(&tq, qkv, (uint64_t)B * S, rs, rs, 128, 64);
  if (r) return r;
  CUtensorMap tq64, tdo64;   // 64-row boxes: Q and dO arrive per query half
  r = make_tmap_bf16_2d(&tq64, qkv, (uint64_t)B * S, rs, rs, 64, 64);
  if (r) return r;
  r = make_tmap_bf16_2d(&tdo64, d_out, (uint64_t)B * S, (uint64_t)nq * d, (uint64_t)nq * d, 64, 64);
  if (r) return r;
  r = make_tmap_f32_2d(&tdq, img, (uint64_t)B * S, rs, rs, 128, 32);
  if (r) return r;
  const float scale = 1.f / sqrtf((float)d);
  const int hpc = bwd_heads_per_cta(S / 128, n_kv, g, B);
  const dim3 grid(S / 128 * (nq / hpc), B);
  if (d == 64) {
    static bool set = false;
    if (!set) { cudaFuncSetAttribute(flash_bwd64_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Bwd64Smem::kTotal); set = true; }
    flash_bwd64_kernel<<<grid, kBwd64Threads, Bwd64Smem::kTotal, stream>>>(tq, tq64, tdo64, tdq, lse2, delta, S, n_kv, g, hpc, scale,
                                                                        scale * 1.4426950408889634f, status, g_bwd_dbg);
  } else {
    static bool set = false;
    if (!set) { cudaFuncSetAttribute(flash_bwd128_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Bwd128Smem::kTotal); set = true; }
    flash_bwd128_kernel<<<grid, kBwd128Threads, Bwd128Smem::kTotal, stream>>>(
        tq, tq64, tdo64, tdq, img, lse2, delta, S, n_kv, g, hpc, scale, scale * 1.4426950408889634f, status);
  }
  if (cudaGetLastError() != cudaSuccess) return -21;
  size_t items = (size_t)B * S * n_kv * (g + 2) * (d / 16);
  int blocks = (int)((items + 255) / 256);
  if (blocks > 148 * 16) blocks = 148 * 16;
  dqkv_finalize_kernel<<<blocks, 256, 0, stream>>>(img, (__nv_bfloat16*)dqkv, rope_table, B * S, S, n_kv, g, d);
  return cudaGetLastError() == cudaSuccess ? 0 : -21;
}

}  // extern "C"
