// Backward triangle attention for sm_100a: dQ, dK, dV and dBias, the work of the reference's
// `_attn_bwd` (flash_tt_attn.py:442-550) with each score tile visited ONCE (5 MMAs and one
// exp2 per score instead of the reference's two passes).
//
// A CTA owns one key block `kb` of one (b,h) and the r-th of NP nearly equal blocks of consecutive
// L1 rows, which it walks in groups of G rows. For each group it keeps K/V of the G
// rows in shared memory and dK/dV of the G rows in TMEM, and walks the query blocks `jb`
// (outer) and the G rows (inner). Per 128 x 128 tile:
//
//   S^T  = K Q^T + c / (scale log2e), dP^T = V dO^T - delta     (tcgen05, operands in smem; c = -(max log2e + log2 sum))
//   P^T  = exp2(S^T*scale*log2e + bias^T*log2e),  dS^T = P^T * dP^T                          (CUDA cores)
//   dV  += P^T dO, dK += dS^T Q                        (A operand read from TMEM)
//   dQ   = dS K                                        (dS staged in smem, M-major)
//
// Two compute warpgroups own one 64-query half of every tile each (thread = key row). S^T and dP^T of a half are
// there together, so one pass forms P and dS without keeping P, and a half has ONE hand-over per tile (its
// dV and dK, and the S^T and dP^T of its next tile, issued back to back). The halves run at their own pace:
// the latency of one's hand-over, barriers and dBias flushes passes behind the other one's arithmetic.
// One warp issues the MMAs of both halves in a fixed order, so the sums in dK and dV are bit-reproducible.
// What leaves the CTA has warps of its own: a drain warpgroup takes dQ and dK / dV out of TMEM, one warp
// sends the dBias boxes.
// The bias is read from a transposed copy (key-major) so that the thread that owns a key row reads its query
// columns with 16-byte shared-memory loads.
//
// dBias: each thread owns one key column and 64 query rows of the (jb,kb) tile and sums dS
// (float32, before rounding) over the G rows in registers. At the end of a query block a half parks its sums as
// two 16 KB boxes (32 queries each): one in the half bias stage that it has just used up (a thread overwrites only
// the bias row that it alone has read), one in a spare buffer. The box warp adds them to the CTA's PRIVATE
// float32 plane (plane index r, key-major) with TMA tile reductions while the compute warps go on. A plane element is
// only ever touched by one CTA, one addition per group, each completed before the next, so the result is
// bit-exact run to run; the planes are summed in fixed order by the finalise kernel.
// dQ leaves the CTA the same way: TMEM -> shared memory -> TMA reduction into a zero-initialised
// float32 buffer (sum over key blocks). With a single key block (L2 <= 128) there is nothing to add up: dQ is scaled,
// rounded and stored like dK and dV, and neither zero fill nor finalisation is needed. Whatever the route (TMA or register stores, tiles or contiguous), an SM
// gets out 32 bytes per cycle of stores and 25 of float32 reductions (30 and 24 with all SMs at it): at D = 32 a tile's
// 16 KB of dQ and third of 64 KB of dBias need 1 560 cycles, at D = 64 32 KB and 64 KB need 4 100.
//
// Measured (whole backward pass, us, before -> with the statistics in the accumulators, the bias loaded a chunk ahead and
// more registers for the service warps): B1 H4 bf16 L768 1 708 -> 1 641, L512 574 -> 546 (fp16 558 -> 533), B4 H8 L256 fp16 671 ->
// 662, B2 H8 L160 204 -> 200; D 64: L512 1 019 -> 1 000, B4 H8 L256 1 330 -> 1 321.
// What bounds it (clock stamps of one CTA, L768 D32, 3 700 cycles a tile): both halves are in their pass together for
// 2 600 cycles, then wait for the issuer, 600 cycles a half for dV, dK and the next S^T, dP^T, of which 430 are the MMAs
// themselves (probe: an MMA with M = 128, K = 16 and A in shared memory takes 48 cycles up to N = 64 and 65 at N = 128;
// with A in TMEM 29 at N = 32). The pass alone takes 1 400 (two warps per scheduler) and 1 900 to 2 000 while the tensor
// core reads its operands from shared memory, which delays the pass's own accesses there; MMAs with A in TMEM do not. The
// rest is instruction fetch: all roles together run through more code than the SM's instruction cache holds (6.6 % of the
// requests miss, 66 % of the peak rate of the next level), so every role's code counts: a second copy of the poll
// in each wait made the whole pass 15 % slower.
// Tried: the four quarters with a hand-over each (768 threads, 96 registers): the issuer, at a good 1 000 cycles per
// turn, became the bound (3.18 ms at L768 against 2.71); 16 queries per TMEM load instead of 8: equal; all of a row's bias
// loaded before the pass (1 724 us against 1 664 for the pass at L768), the issuer's MMAs in loops instead of unrolled
// (2 001), its other barriers polled together ahead of the hand-over (1 781), records for 32 queries at a time (2 240),
// 200 registers for the compute warps and 56 for the others (1 891).
//
//   warp 0      : tcgen05 issuer (lowest warp id: the scheduler prefers older warps)
//   warp 1      : TMA producer        warp 2 : statistics records        warp 3 : dBias boxes (TMA reductions)
//   warps 4-7   : drain warpgroup (dQ tiles, finished dK / dV rows)
//   warps 8-15  : two compute warpgroups, one 64-query half of the tile each
// Producer and issuer loops run warp-uniformly; one elected lane issues the TMA / MMA.
#include "fta_kernels.h"
#include "tc05.cuh"

namespace fta {
namespace {

constexpr float kLog2e = 1.4426950408889634f;
constexpr int kBwdThreads = 512;
// registers per thread after setmaxnreg: 2 * 176 + 72 + 88 = 4 * 128, the block's allotment at launch. The service warps
// (issuer) spill with less than 88.
constexpr int kRegsCompute = 176, kRegsDrain = 72, kRegsService = 88;

template <int kD>
struct BwdCfg {
  static constexpr int G = (kD == 32) ? 3 : 1;   // rows per group (TMEM: 256 + 2*D + 2*D*G <= 512)
  static constexpr int NQ = 2;                   // Q/dO ring depth (in tiles; a slot's halves come and go by themselves)
  static constexpr int NX = (kD == 32) ? 2 : 1;  // spare 16 KB boxes for dBias: one per query half, or one in turns
  // K/V of the next group's first row are there before this group ends (its slot was freed G - 1 tiles ago)
  static constexpr bool KV_AHEAD = G >= 3;
  static constexpr int DQS_B = 128 * 16 * 4;  // dQ staging tile: 128 queries x 16 columns, float32
  static constexpr int TILE_B = 128 * kD * 2;
  static constexpr int STAGE_B = 2 * TILE_B + 2048;  // Q, dO, a 16-byte record of statistics per query
  static constexpr int BIAS_B = 128 * 128 * 2;
  static constexpr int DS_B = 128 * 128 * 2;
  static constexpr int OFF_KV = 0;
  static constexpr int OFF_QDO = OFF_KV + G * 2 * TILE_B;
  static constexpr int OFF_BIAS = OFF_QDO + NQ * STAGE_B;
  static constexpr int OFF_DS = OFF_BIAS + 2 * BIAS_B;
  static constexpr int OFF_DQS = OFF_DS + DS_B;
  static constexpr int OFF_BOX = OFF_DQS + DQS_B;
  static constexpr int OFF_ONES = OFF_BOX + NX * 16384;  // A operands that pick c / -delta from the records: 2 x 128 rows x 8
  static constexpr int OFF_ZERO = OFF_ONES + 4096;       // 64 x 8 zeros: the upper half of a record's K = 16
  static constexpr int OFF_BAR = OFF_ZERO + 1024;
  static constexpr int B_KVFULL = 0;                  // per row of the group
  static constexpr int B_KVFREE = B_KVFULL + G;
  static constexpr int B_QDOFULL = B_KVFREE + G;      // 2 * ring slot + query half
  static constexpr int B_QDOEMPTY = B_QDOFULL + 2 * NQ;
  static constexpr int B_BIASFULL = B_QDOEMPTY + 2 * NQ;  // 2 * stage + half
  static constexpr int B_BIASEMPTY = B_BIASFULL + 4;
  static constexpr int B_XFULL = B_BIASEMPTY + 4;     // per half: S^T and dP^T of its next tile are in TMEM
  static constexpr int B_UFULL = B_XFULL + 2;         // per half: its four warps have written P^T and dS^T
  static constexpr int B_DQDONE = B_UFULL + 2;        // per dQ buffer (a single barrier could run a phase ahead of the drain)
  static constexpr int B_DQFREE = B_DQDONE + 2;       // the drain warpgroup has copied the buffer out
  static constexpr int B_ACCFULL = B_DQFREE + 2;      // per row of the group: dK / dV complete
  static constexpr int B_ACCFREE = B_ACCFULL + G;
  static constexpr int B_BOX = B_ACCFREE + G;         // dBias, per half: both boxes of a query block are parked
  static constexpr int B_BOXFREE = B_BOX + 2;         // per half: the spare box it parked has been read
  static constexpr int NBAR = B_BOXFREE + 2;
  static constexpr int SMEM_BYTES = OFF_BAR + NBAR * 8 + 16 + 1024;  // + tmem slot / abort flag + alignment slack
  static constexpr uint64_t SWZ = (kD == 32) ? kSwz64 : kSwz128;
  static constexpr uint32_t ROW_B = kD * 2;
  static constexpr uint32_t SBO = 8 * ROW_B;
  static constexpr uint32_t HALF_B = 64 * ROW_B;     // bytes of 64 queries of a Q / dO tile
  // TMEM columns
  static constexpr uint32_t TM_ST = 0;               // half h: 64 columns at TM_ST + 64 h; P^T over the first 32
  static constexpr uint32_t TM_DP = 128;
  static constexpr uint32_t TM_DQ = 256;             // two dQ buffers of kD columns
  static constexpr uint32_t TM_ACC = 256 + 2 * kD;   // dK_g at TM_ACC + g*2*kD, dV_g right after
  static_assert(TM_ACC + G * 2 * kD <= 512, "TMEM budget");
};

struct BwdParams {
  const float* lse;  // three planes: -max (natural-log units), -log2(sum), c (see the forward kernel)
  const float* delta;
  int* status;
  int H, L1, L2, NP, BH;
  int stat_pitch;  // row pitch of lse / delta: L2 rounded up to 128
  float scale;  // sm_scale
  long long stat_stride;  // elements between the statistics planes
};

// Two numbers as three bfloat16 each (24 bits and more), as the six leading elements of a query's record
__device__ __forceinline__ uint4 stat_record(float c, float d, uint32_t flags) {
  const uint32_t h = pack_bf16x2(c, d);
  c -= __uint_as_float(h << 16);
  d -= __uint_as_float(h & 0xFFFF0000u);
  const uint32_t m = pack_bf16x2(c, d);
  c -= __uint_as_float(m << 16);
  d -= __uint_as_float(m & 0xFFFF0000u);
  const uint32_t l = pack_bf16x2(c, d);
  return make_uint4(__byte_perm(h, m, 0x5410), __byte_perm(l, h, 0x7610), __byte_perm(m, l, 0x7632), flags);
}

template <int kD, bool kBf16>
__global__ void __launch_bounds__(kBwdThreads, 1)
fta_bwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
               const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmDO,
               const __grid_constant__ CUtensorMap tmBiasT, const __grid_constant__ CUtensorMap tmDQ,
               const __grid_constant__ CUtensorMap tmPlane, const __grid_constant__ CUtensorMap tmDK,
               const __grid_constant__ CUtensorMap tmDV, const __grid_constant__ CUtensorMap tmDQ16, const BwdParams p) {
  using C = BwdCfg<kD>;
  constexpr int G = C::G;
  extern __shared__ uint8_t smem_raw[];
  // 1 KB alignment by an offset from the shared array itself, so that the compiler keeps the
  // shared address space (ld.shared / st.shared instead of generic accesses)
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint8_t* sKV = smem + C::OFF_KV;      // [g][K tile | V tile]
  uint8_t* sQDO = smem + C::OFF_QDO;    // [slot][Q | dO | statistics]
  uint8_t* sBias = smem + C::OFF_BIAS;  // [stage][query half][key row][64 queries], 128B swizzle
  uint8_t* sDS = smem + C::OFF_DS;      // [query half][key row][64 queries], 128B swizzle
  uint8_t* sDQ = smem + C::OFF_DQS;     // float32 dQ tile on its way to the TMA reduction
  uint8_t* sBox = smem + C::OFF_BOX;
  uint8_t* sOnes = smem + C::OFF_ONES;
  uint8_t* sZero = smem + C::OFF_ZERO;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::OFF_BAR);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + C::NBAR);
  int* abort_flag = reinterpret_cast<int*>(tmem_slot + 1);
  const uint32_t bar0 = smem_u32(bars);
  auto bar = [&](int i) { return bar0 + 8u * static_cast<uint32_t>(i); };

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // a ragged last block (L2 not a multiple of 128) is padded: loads fill zeros, the key-major bias
  // copy holds -inf for keys past L2, the statistics give P = 0 for queries past L2, stores are clipped
  const int nkb = (p.L2 + 127) / 128, nq = nkb;
  const int kb = blockIdx.x % nkb;
  const int r = (blockIdx.x / nkb) % p.NP;
  const int bh = blockIdx.x / (nkb * p.NP);
  const int b = bh / p.H, h = bh % p.H;
  // This CTA's rows: the r-th of NP nearly equal blocks of consecutive L1 rows (sizes differ by at
  // most one row, none empty since NP <= L1), walked in groups of G rows with a short last group.
  const int row_begin = static_cast<int>(static_cast<long long>(r) * p.L1 / p.NP);
  const int row_end = static_cast<int>(static_cast<long long>(r + 1) * p.L1 / p.NP);
  const int ngroups = (row_end - row_begin + G - 1) / G;
  const WaitCtx w{smem_u32(abort_flag), p.status};

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int i = 0; i < G; ++i) {
      mbar_init(bar(C::B_KVFULL + i), 1);
      mbar_init(bar(C::B_KVFREE + i), 1);
      mbar_init(bar(C::B_ACCFULL + i), 1);
      mbar_init(bar(C::B_ACCFREE + i), 4);
    }
    for (int i = 0; i < 2 * C::NQ; ++i) {
      mbar_init(bar(C::B_QDOFULL + i), 2);  // the producer's expected bytes, the record warp
      mbar_init(bar(C::B_QDOEMPTY + i), 1);
    }
    for (int i = 0; i < 4; ++i) {
      mbar_init(bar(C::B_BIASFULL + i), 1);
      mbar_init(bar(C::B_BIASEMPTY + i), 1);  // box warp, once the box parked in the half stage is read
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(bar(C::B_DQDONE + i), 1);
      mbar_init(bar(C::B_DQFREE + i), 4);
      mbar_init(bar(C::B_XFULL + i), 1);
      mbar_init(bar(C::B_UFULL + i), 4);  // one arrive per warp of the half
      mbar_init(bar(C::B_BOX + i), 4);
      mbar_init(bar(C::B_BOXFREE + i), 1);
    }
    mbar_fence_init();
  }
  if (threadIdx.x < 256) {
    reinterpret_cast<uint4*>(sOnes)[threadIdx.x] = threadIdx.x < 128 ? make_uint4(0x3F803F80u, 0x00003F80u, 0u, 0u)   // 1 1 1 0 0 0 0 0
                                                                     : make_uint4(0u, 0xBF800000u, 0xBF80BF80u, 0u);  // 0 0 0 -1 -1 -1 0 0
    if (threadIdx.x < 64) reinterpret_cast<uint4*>(sZero)[threadIdx.x] = make_uint4(0u, 0u, 0u, 0u);
    fence_proxy_async_smem();
  }
  if (warp == 0) {
    tmem_alloc(smem_u32(tmem_slot), 512);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tbase = *tmem_slot;

  if (warp < 4) {
    reg_dec<kRegsService>();
    if (warp == 1) {
      // ---------------------------------------------------------------- TMA producer
      if (elect_one()) {
        tma_prefetch_desc(&tmQ);
        tma_prefetch_desc(&tmK);
        tma_prefetch_desc(&tmV);
        tma_prefetch_desc(&tmDO);
        tma_prefetch_desc(&tmBiasT);
        tma_prefetch_desc(&tmDQ);
        tma_prefetch_desc(&tmPlane);
        tma_prefetch_desc(&tmDK);
        tma_prefetch_desc(&tmDV);
      }
      // K/V/Q/dO tiles stream through L2 (each is read within a short window and never again);
      // the bias tiles are re-read by every group and stay
      const uint64_t pol_stream = l2_policy_evict_first(), pol_keep = l2_policy_evict_last();
      bool ok = true;
      int s = 0, nb = 0;
      uint32_t ring_par = 1;  // of the wait for an empty slot
      for (int n = 0; n < ngroups && ok; ++n) {
        const int i0 = row_begin + n * G;
        const int Gc = min(G, row_end - i0);
        for (int jb = 0; jb < nq && ok; ++jb, ++nb) {
          for (int g = 0; g < Gc; ++g) {
            if (jb == 0) {
              ok = mbar_wait_warp(bar(C::B_KVFREE + g), (n & 1) ^ 1, w, 0x21);
              if (!ok) break;
              if (elect_one()) {
                mbar_expect_tx(bar(C::B_KVFULL + g), 2 * C::TILE_B);
                tma_load_5d_hint(smem_u32(sKV + g * 2 * C::TILE_B), &tmK, bar(C::B_KVFULL + g), 0, kb * 128, i0 + g, h, b,
                                 pol_stream);
                tma_load_5d_hint(smem_u32(sKV + g * 2 * C::TILE_B + C::TILE_B), &tmV, bar(C::B_KVFULL + g), 0, kb * 128,
                                 i0 + g, h, b, pol_stream);
                // K/V of the next group are read by no other CTA: bring them into L2 a whole group ahead
                const int i1 = i0 + G + g;
                if (i1 < row_end) {
                  tma_prefetch_l2_5d(&tmK, 0, kb * 128, i1, h, b);
                  tma_prefetch_l2_5d(&tmV, 0, kb * 128, i1, h, b);
                }
              }
              __syncwarp();
            }
#pragma unroll 1
            for (int hf = 0; hf < 2 && ok; ++hf) {
              ok = mbar_wait_warp(bar(C::B_QDOEMPTY + 2 * s + hf), ring_par, w, 0x23);
              if (!ok) break;
              if (elect_one()) {
                const uint32_t st = smem_u32(sQDO + s * C::STAGE_B);
                const uint32_t full = bar(C::B_QDOFULL + 2 * s + hf);
                const int q0 = jb * 128 + hf * 64;
                mbar_expect_tx(full, C::TILE_B);
                tma_load_5d_hint(st + hf * C::HALF_B, &tmQ, full, 0, q0, i0 + g, h, b, pol_stream);
                tma_load_5d_hint(st + C::TILE_B + hf * C::HALF_B, &tmDO, full, 0, q0, i0 + g, h, b, pol_stream);
              }
              __syncwarp();
              if (g == 0) {  // after the Q/dO loads: the half stages come free later than the ring slot
                const int bs = 2 * (nb & 1) + hf;
                ok = mbar_wait_warp(bar(C::B_BIASEMPTY + bs), ((nb >> 1) & 1) ^ 1, w, 0x22);
                if (!ok) break;
                if (elect_one()) {
                  // transposed bias: innermost coordinate = query, then key
                  mbar_expect_tx(bar(C::B_BIASFULL + bs), C::BIAS_B / 2);
                  tma_load_4d_hint(smem_u32(sBias + bs * 16384), &tmBiasT, bar(C::B_BIASFULL + bs), jb * 128 + hf * 64,
                                   kb * 128, h, b, pol_keep);
                }
                __syncwarp();
              }
            }
            if (!ok) break;
            if (++s == C::NQ) {
              s = 0;
              ring_par ^= 1u;
            }
          }
        }
      }
    } else if (warp == 0) {
      // ---------------------------------------------------------------- MMA issuer
      // One hand-over per tile and half: when a half has written P^T and dS^T of tile t, its dV and dK
      // and the S^T and dP^T of its next tile are issued back to back. The other half computes meanwhile.
      // A tile whose predecessor could not look ahead (the first one; with a single K/V slot, the first one of
      // a row) starts afresh. The very first one starts half 1 when half 0 has done its part, so that the halves
      // work in turns; with a restart per row that would cost more than it gives.
      // This warp is on every half's critical path: operands are checked and descriptors built BEFORE
      // the wait for the half, so that a hand-over is poll, fence, MMAs.
      constexpr int fmt = kBf16 ? 1 : 0;
      constexpr uint32_t idesc_acc = umma_idesc_f16(fmt, 128, kD, 0, 1);  // dV, dK (A in TMEM, B M-major)
      constexpr uint32_t idesc_x = umma_idesc_f16(fmt, 128, 64, 0, 0);    // S^T, dP^T: 64 queries
      constexpr uint32_t idesc_st = umma_idesc_f16(1, 128, 64, 0, 0);     // the records' part of S^T, dP^T: bfloat16
      constexpr uint32_t idesc_dq = umma_idesc_f16(fmt, 128, kD, 1, 1);   // dQ (A, B M-major)
      // Descriptors as 32-bit low words (address and leading-dimension offset); the high word is a constant.
      constexpr uint32_t HI = (C::SBO >> 4) | (1u << 14) | (static_cast<uint32_t>(C::SWZ) << 29);
      auto mk = [](uint32_t lo) { return (static_cast<uint64_t>(HI) << 32) | lo; };
      constexpr uint32_t LK = 1u << 16, LM = (C::SBO >> 4) << 16;  // K-major: lbo = 16 bytes; M-major: lbo = SBO
      constexpr uint32_t KSTEP = (2 * C::SBO) >> 4;                // 16 rows further (M-major operand)
      const uint32_t lo_kv = smem_u32(sKV) >> 4, lo_qdo = smem_u32(sQDO) >> 4;  // shared addresses are below 2^18
      constexpr uint32_t KV_STEP = 2 * C::TILE_B >> 4, SLOT_STEP = C::STAGE_B >> 4, TILE_STEP = C::TILE_B >> 4,
                         HALF_STEP = C::HALF_B >> 4, REC_OFF = 2 * C::TILE_B >> 4, REC_HALF = 1024 >> 4;
      bool ok = true, fresh = true;
      int n = 0, jb = 0, g = 0, Gc = min(G, row_end - row_begin), slot = 0, tt = 0;
      uint32_t ring_par = 0;
      // The records: rows of 8 elements without a swizzle, 128 bytes per 8 rows; the upper half of K = 16 is zeros on their
      // side (and whatever finite numbers follow on the other). LBO = distance to it.
      constexpr uint32_t HI_ST = (128u >> 4) | (1u << 14);
      auto mk_st = [](uint32_t lo) { return (static_cast<uint64_t>(HI_ST) << 32) | lo; };
      const uint32_t lo_ones = (smem_u32(sOnes) >> 4) | (128u >> 4) << 16, lo_zero = smem_u32(sZero) >> 4;
      // S^T = K Q^T + c / (scale log2 e), dP^T = V dO^T - delta of half hf, by the elected lane; kv, q, st: low words of K, of
      // the half's Q and of its records
      auto issue_x = [&](int hf, uint32_t kv, uint32_t q, uint32_t st) {
        const uint64_t rec = mk_st(st | (lo_zero - st) << 16);
        umma_ss(tbase + C::TM_ST + hf * 64, mk_st(lo_ones), rec, idesc_st, 0);
#pragma unroll
        for (int ks = 0; ks < kD / 16; ++ks)
          umma_ss(tbase + C::TM_ST + hf * 64, mk(kv | LK) + ks * 2, mk(q | LK) + ks * 2, idesc_x, 1);
        umma_ss(tbase + C::TM_DP + hf * 64, mk_st(lo_ones + (2048 >> 4)), rec, idesc_st, 0);
#pragma unroll
        for (int ks = 0; ks < kD / 16; ++ks)
          umma_ss(tbase + C::TM_DP + hf * 64, mk((kv + TILE_STEP) | LK) + ks * 2, mk((q + TILE_STEP) | LK) + ks * 2, idesc_x, 1);
        umma_commit(bar(C::B_XFULL + hf));
      };
      auto start_half1 = [&]() -> bool {
        ok = mbar_wait_warp(bar(C::B_QDOFULL + 2 * slot + 1), ring_par, w, 0x35);
        if (!ok) return false;
        tc_fence_after_sync();
        if (elect_one()) issue_x(1, lo_kv + g * KV_STEP, lo_qdo + slot * SLOT_STEP + HALF_STEP, lo_qdo + slot * SLOT_STEP + REC_OFF + REC_HALF);
        __syncwarp();
        return true;
      };
      while (ok) {
        if (fresh) {
          ok = mbar_wait_warp(bar(C::B_KVFULL + g), n & 1, w, 0x32) &&
               mbar_wait_warp(bar(C::B_QDOFULL + 2 * slot), ring_par, w, 0x30);
          if (!ok) break;
          tc_fence_after_sync();
          if (elect_one()) issue_x(0, lo_kv + g * KV_STEP, lo_qdo + slot * SLOT_STEP, lo_qdo + slot * SLOT_STEP + REC_OFF);
          __syncwarp();
          if (!C::KV_AHEAD && !start_half1()) break;
        }
        // the tile after this one
        int n1 = n, jb1 = jb, g1 = g + 1, Gc1 = Gc, slot1 = slot + 1;
        uint32_t ring_par1 = ring_par;
        if (g1 == Gc) {
          g1 = 0;
          if (++jb1 == nq) {
            jb1 = 0;
            ++n1;
            Gc1 = min(G, row_end - (row_begin + n1 * G));
          }
        }
        if (slot1 == C::NQ) {
          slot1 = 0;
          ring_par1 ^= 1u;
        }
        const bool cont = n1 < ngroups && (C::KV_AHEAD || n1 == n);  // its S^T and dP^T are issued from this one
        const bool last = jb == nq - 1;
        const uint32_t acc = tbase + C::TM_ACC + g * 2 * kD;
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
          const uint32_t qv = lo_qdo + slot * SLOT_STEP + hf * HALF_STEP;
          const uint32_t kvn = lo_kv + g1 * KV_STEP, qn = lo_qdo + slot1 * SLOT_STEP + hf * HALF_STEP;
          const uint32_t stn = lo_qdo + slot1 * SLOT_STEP + REC_OFF + hf * REC_HALF;
          const uint32_t first = (hf || jb > 0) ? 1u : 0u;  // 0: the accumulators start at zero
          asm volatile("" ::"r"(qv), "r"(kvn), "r"(qn), "r"(stn), "r"(first));
          if (cont) {
            ok = mbar_wait_warp(bar(C::B_QDOFULL + 2 * slot1 + hf), ring_par1, w, 0x31);
            if (ok && hf == 0 && jb1 == 0) ok = mbar_wait_warp(bar(C::B_KVFULL + g1), n1 & 1, w, 0x36);
          }
          if (ok && hf == 0 && jb == 0 && n > 0) ok = mbar_wait_warp(bar(C::B_ACCFREE + g), (n - 1) & 1, w, 0x34);
          if (ok) ok = mbar_wait_warp(bar(C::B_UFULL + hf), tt & 1, w, 0x33);
          if (!ok) break;
          tc_fence_after_sync();
          if (elect_one()) {
            // dV += P^T dO, dK += dS^T Q
#pragma unroll
            for (int ks = 0; ks < 4; ++ks)
              umma_ts(acc + kD, tbase + C::TM_ST + hf * 64 + ks * 8, mk((qv + TILE_STEP) | LM) + ks * KSTEP, idesc_acc,
                      ks > 0 ? 1u : first);
#pragma unroll
            for (int ks = 0; ks < 4; ++ks)
              umma_ts(acc, tbase + C::TM_DP + hf * 64 + ks * 8, mk(qv | LM) + ks * KSTEP, idesc_acc, ks > 0 ? 1u : first);
            if (cont) issue_x(hf, kvn, qn, stn);
            umma_commit(bar(C::B_QDOEMPTY + 2 * slot + hf));
            if (hf == 1 && last) umma_commit(bar(C::B_ACCFULL + g));
          }
          __syncwarp();
          if (C::KV_AHEAD && hf == 0 && fresh && !start_half1()) break;
        }
        if (!ok) break;
        // dQ = dS K, behind everything that a half waits for; its TMEM buffer was drained a tile ago
        if (tt >= 2) ok = mbar_wait_warp(bar(C::B_DQFREE + (tt & 1)), ((tt >> 1) & 1) ^ 1, w, 0x3e);
        if (!ok) break;
        tc_fence_after_sync();
        if (elect_one()) {
          const uint64_t dSm = umma_smem_desc(smem_u32(sDS), 16384, 1024, kSwz128);
#pragma unroll
          for (int ks = 0; ks < 8; ++ks)
            umma_ss(tbase + C::TM_DQ + (tt & 1) * kD, dSm + ks * (2048 >> 4), mk((lo_kv + g * KV_STEP) | LM) + ks * KSTEP,
                    idesc_dq, ks > 0);
          umma_commit(bar(C::B_DQDONE + (tt & 1)));
          if (last) umma_commit(bar(C::B_KVFREE + g));
        }
        __syncwarp();
        if (n1 == ngroups) break;
        fresh = !cont;
        n = n1;
        jb = jb1;
        g = g1;
        Gc = Gc1;
        slot = slot1;
        ring_par = ring_par1;
        ++tt;
      }
    } else if (warp == 2) {
      // ---------------------------------------------------------------- record warp
      // c / (scale log2 e) and delta of a query as three bfloat16 each, in 16 bytes: one K = 16 step of the tensor core with
      // rows of ones adds the first to all of the query's S^T, one with rows of minus ones takes the second from all of its
      // dP^T. As operands of the pass they would be broadcast loads, and every 16 bytes a thread loads from shared memory
      // take its port for four cycles per warp, broadcast or not: 1 024 of a tile's 3 800.
      // A query whose numbers do not go into a record (|c| > 256, where three rounded additions would cost P more than
      // they do here; infinite or NaN) is flagged and left out; the compute warps then see to it themselves.
      const float inv_k1 = 1.0f / (p.scale * kLog2e);
      const float* cp = p.lse + 2 * p.stat_stride;
      float2 cn[2], dn[2];
      auto fetch = [&](int i, int jb) {
        const long long off = (static_cast<long long>(bh) * p.L1 + i) * p.stat_pitch + jb * 128 + 2 * lane;
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
          cn[hf] = __ldg(reinterpret_cast<const float2*>(cp + off + hf * 64));
          dn[hf] = __ldg(reinterpret_cast<const float2*>(p.delta + off + hf * 64));
        }
      };
      bool ok = true;
      int s = 0;
      uint32_t ring_par = 1;
      fetch(row_begin, 0);
      for (int n = 0; n < ngroups && ok; ++n) {
        const int i0 = row_begin + n * G;
        const int Gc = min(G, row_end - i0);
        for (int jb = 0; jb < nq && ok; ++jb) {
          for (int g = 0; g < Gc; ++g) {
            const float2 cv[2] = {cn[0], cn[1]}, dv[2] = {dn[0], dn[1]};
            const bool wrap_g = g + 1 == Gc, wrap_jb = wrap_g && jb + 1 == nq;
            const int i1 = wrap_jb ? i0 + G : wrap_g ? i0 : i0 + g + 1;
            if (i1 < row_end) fetch(i1, wrap_jb ? 0 : wrap_g ? jb + 1 : jb);
#pragma unroll 1
            for (int hf = 0; hf < 2; ++hf) {
              const float2 c = hf ? cv[1] : cv[0], d = hf ? dv[1] : dv[0];
              // an empty row (c = -inf) needs P = 0 only
              float cx = c.x < -1.0e30f ? -1.0e30f : c.x, cy = c.y < -1.0e30f ? -1.0e30f : c.y;
              const bool bigx = !(fabsf(cx) <= 256.f || cx == -1.0e30f), bigy = !(fabsf(cy) <= 256.f || cy == -1.0e30f);
              cx *= inv_k1;
              cy *= inv_k1;
              const bool fx = bigx || !(fabsf(cx) < 1.0e37f) || !(fabsf(d.x) < 1.0e37f);
              const bool fy = bigy || !(fabsf(cy) < 1.0e37f) || !(fabsf(d.y) < 1.0e37f);
              const uint32_t any = __any_sync(0xffffffffu, fx || fy) && lane == 0 ? 0x3F800000u : 0u;
              const uint4 rx = stat_record(fx ? 0.f : cx, fx ? 0.f : d.x, (fx ? 0x3F80u : 0u) | any);
              const uint4 ry = stat_record(fy ? 0.f : cy, fy ? 0.f : d.y, fy ? 0x3F80u : 0u);
              ok = mbar_wait_warp(bar(C::B_QDOEMPTY + 2 * s + hf), ring_par, w, 0x24);
              if (!ok) break;
              const uint32_t dst = smem_u32(sQDO + s * C::STAGE_B) + 2 * C::TILE_B + hf * 1024 + lane * 32;
              st_shared_v4(dst, rx.x, rx.y, rx.z, rx.w);
              st_shared_v4(dst + 16, ry.x, ry.y, ry.z, ry.w);
              fence_proxy_async_smem();
              __syncwarp();
              if (lane == 0) mbar_arrive(bar(C::B_QDOFULL + 2 * s + hf));
            }
            if (!ok) break;
            if (++s == C::NQ) {
              s = 0;
              ring_par ^= 1u;
            }
          }
        }
      }
    } else if (warp == 3) {
      // ---------------------------------------------------------------- dBias box warp
      // The boxes parked by the compute halves (two of 128 keys x 32 queries each), each added to (first group: stored
      // into) this CTA's private key-major plane.
      // The planes (a few tens of MB, added to once per group) must stay in L2 between groups: with
      // default priority the dQ stream evicts them and every addition becomes a DRAM read + write.
      const uint64_t pol_keep = l2_policy_evict_last();
      const int pkey = kb * 128, pidx = r * p.BH + bh;  // first key row of this CTA's tile, its plane
      bool ok = true;
      int nb = 0;
      for (int n = 0; n < ngroups && ok; ++n) {
        for (int jb = 0; jb < nq && ok; ++jb, ++nb) {
#pragma unroll 1
          for (int hf = 0; hf < 2; ++hf) {
            const int bs = 2 * (nb & 1) + hf, x = hf & (C::NX - 1);
            ok = mbar_wait_warp(bar(C::B_BOX + hf), nb & 1, w, 0x51);
            if (!ok) break;
            if (elect_one()) {
              // The elements that these boxes are added to were last written a group ago, nq query blocks of four
              // boxes back: with all but the newest two of this thread's transfers complete, they are.
              if (n > 0) bulk_wait_le<2>();
#pragma unroll 1
              for (int box = 0; box < 2; ++box) {
                const uint32_t src = box ? smem_u32(sBox + x * 16384) : smem_u32(sBias + bs * 16384);
                const int qcol = jb * 128 + hf * 64 + box * 32;
                if (n == 0) tma_store_3d_hint(&tmPlane, src, qcol, pkey, pidx, pol_keep);
                else tma_reduce_add_3d_hint(&tmPlane, src, qcol, pkey, pidx, pol_keep);
                bulk_commit_group();
              }
              bulk_wait_read_le<1>();
              mbar_arrive(bar(C::B_BIASEMPTY + bs));
              bulk_wait_read_all();
              mbar_arrive(bar(C::B_BOXFREE + hf));
            }
            __syncwarp();
          }
        }
      }
      if (elect_one()) bulk_wait_all();
      __syncwarp();
    }
  } else if (warp < 8) {
    // ------------------------------------------------------------------ drain warpgroup
    // Takes finished results out of TMEM: each dQ tile (to a staging tile in shared memory and from there, 32 query
    // rows per warp, into the float32 accumulator with TMA reductions), and dK / dV of a row after its
    // last query block. Every warp handles its own 32 TMEM lanes from end to end, so the four need no barrier.
    reg_dec<kRegsDrain>();
    const uint32_t lane_off = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const int row0 = (warp & 3) * 32;  // first TMEM lane: query row of a dQ tile, key row of dK / dV
    const uint32_t stage = smem_u32(sDQ) + (warp & 3) * 2048;
    // 32 columns of this warp's 32 rows, scaled and rounded, through the staging rows (64-byte swizzle) to a box of an
    // output tensor, clipped by its map. Not from registers: stores that find the SM's way out full, as it is when
    // dBias boxes are leaving, hold up the shared-memory accesses of the compute warps behind them.
    // `free_bar`: arrived at once TMEM has been read (0: none).
    auto emit = [&](uint32_t taddr, const CUtensorMap* map, int col, int row, int irow, float mul, uint32_t free_bar) {
      uint32_t x[16], pk[16];
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        tmem_ld16(taddr + col + half * 16 + lane_off, x);
        tmem_ld_wait();
#pragma unroll
        for (int e = 0; e < 8; ++e)
          pk[half * 8 + e] = pack2<kBf16>(__uint_as_float(x[2 * e]) * mul, __uint_as_float(x[2 * e + 1]) * mul);
      }
      if (elect_one()) bulk_wait_read_all();  // this warp's previous transfer has read the staging rows
      if (free_bar) tc_fence_before_sync();
      __syncwarp();
      if (free_bar && lane == 0) mbar_arrive(free_bar);
#pragma unroll
      for (int j = 0; j < 4; ++j)
        st_shared_v4(stage + lane * 64 + ((j ^ ((lane >> 1) & 3)) << 4), pk[4 * j], pk[4 * j + 1], pk[4 * j + 2], pk[4 * j + 3]);
      fence_proxy_async_smem();
      __syncwarp();
      if (elect_one()) {
        tma_store_5d(map, stage, col, row, irow, h, b);
        bulk_commit_group();
      }
      __syncwarp();
    };
    bool ok = true;
    int tt = 0;
    for (int n = 0; n < ngroups && ok; ++n) {
      const int i0 = row_begin + n * G;
      const int Gc = min(G, row_end - i0);
      for (int jb = 0; jb < nq && ok; ++jb) {
        for (int g = 0; g < Gc; ++g, ++tt) {
          const int buf = tt & 1;
          ok = mbar_wait_warp(bar(C::B_DQDONE + buf), (tt >> 1) & 1, w, 0x46);
          if (!ok) break;
          tc_fence_after_sync();
          if (nkb == 1) {
#pragma unroll 1
            for (int c = 0; c < kD; c += 32)
              emit(tbase + C::TM_DQ + buf * kD, &tmDQ16, c, row0, i0 + g, p.scale, c + 32 == kD ? bar(C::B_DQFREE + buf) : 0u);
          } else {
#pragma unroll 1
          for (int c = 0; c < kD / 16; ++c) {
            uint32_t qv[16];
            tmem_ld16(tbase + C::TM_DQ + buf * kD + c * 16 + lane_off, qv);
            if (elect_one()) bulk_wait_read_all();  // this warp's previous reduction has read the staging rows
            tmem_ld_wait();
            if (c == kD / 16 - 1) tc_fence_before_sync();
            __syncwarp();
            if (c == kD / 16 - 1 && lane == 0) mbar_arrive(bar(C::B_DQFREE + buf));
#pragma unroll
            for (int j = 0; j < 4; ++j)  // 64-byte swizzle
              st_shared_v4(stage + lane * 64 + ((j ^ ((lane >> 1) & 3)) << 4), qv[4 * j], qv[4 * j + 1], qv[4 * j + 2],
                           qv[4 * j + 3]);
            fence_proxy_async_smem();
            __syncwarp();
            if (elect_one()) {
              tma_reduce_add_3d(&tmDQ, stage, c * 16, jb * 128 + row0, bh * p.L1 + i0 + g);
              bulk_commit_group();
            }
            __syncwarp();
          }
          }
          if (jb == nq - 1) {
            ok = mbar_wait_warp(bar(C::B_ACCFULL + g), n & 1, w, 0x45);
            if (!ok) break;
            tc_fence_after_sync();
#pragma unroll 1
            for (int c = 0; c < 2 * kD; c += 32) {  // dK (scaled by sm_scale, flash_tt_attn.py:518), then dV
              const bool is_dv = c >= kD;
              emit(tbase + C::TM_ACC + g * 2 * kD + (is_dv ? kD : 0), is_dv ? &tmDV : &tmDK, c & (kD - 1), kb * 128 + row0, i0 + g,
                   is_dv ? 1.0f : p.scale, c + 32 == 2 * kD ? bar(C::B_ACCFREE + g) : 0u);
            }
          }
        }
      }
    }
    if (elect_one()) bulk_wait_all();
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ compute warpgroups
    reg_inc<kRegsCompute>();
    const int hf = (warp >> 2) - 2;          // query half
    const int key = (warp & 3) * 32 + lane;  // key row of the block == TMEM lane
    const uint32_t lane_off = static_cast<uint32_t>((warp & 3) * 32) << 16;
    // this half's 64 fp32 columns of S^T / dP^T; P^T / dS^T overwrite the first 32 of them
    const uint32_t tST = tbase + C::TM_ST + hf * 64 + lane_off;
    const uint32_t tDP = tbase + C::TM_DP + hf * 64 + lane_off;
    const uint32_t my_ds = smem_u32(sDS) + hf * 16384 + key * 128;
    bool ok = true;
    int tt = 0, nb = 0, slot = 0;
    uint32_t ring_par = 0;
    uint32_t q_in = 0, b_in = 0;  // early polls: statistics of the next tile, bias of the next query block
    for (int n = 0; n < ngroups && ok; ++n) {
      const int Gc = min(G, row_end - (row_begin + n * G));
      for (int jb = 0; jb < nq && ok; ++jb, ++nb) {
        f32x2 acc[32];  // dBias sums: this key column x 64 query rows
#pragma unroll
        for (int c = 0; c < 32; ++c) acc[c] = mk2(0.f, 0.f);
        const int bs = 2 * (nb & 1) + hf;
        ok = mbar_finish_wait(b_in, bar(C::B_BIASFULL + bs), (nb >> 1) & 1, w, 0x41);
        if (!ok) break;
#pragma unroll 1
        for (int g = 0; g < Gc; ++g, ++tt) {
          ok = mbar_finish_wait(q_in, bar(C::B_QDOFULL + 2 * slot + hf), ring_par, w, 0x43) &&  // statistics visible
               mbar_wait_warp(bar(C::B_XFULL + hf), tt & 1, w, 0x42);
          if (!ok) break;
          tc_fence_after_sync();
          const uint4* recs = reinterpret_cast<const uint4*>(sQDO + slot * C::STAGE_B + 2 * C::TILE_B + hf * 1024);
          const uint8_t* brow = sBias + bs * 16384 + key * 128;
          f32x2 k1_2 = mk2(p.scale * kLog2e, p.scale * kLog2e), log2e2 = mk2(kLog2e, kLog2e);
          if (++slot == C::NQ) {
            slot = 0;
            ring_par ^= 1u;
          }
          // P^T = exp2((S^T*scale + bias^T - max)*log2e - log2 sum) as y = s*(scale*log2e) + b*log2e, with the statistics in s
          // already, unless a query of the half is flagged.
          if (recs[0].w != 0u) {
            // Rare (rows masked with a large negative bias): form y, and dP - delta of the flagged queries, in a pass of its
            // own, in place of S^T and dP^T, and have the pass below take them as they are.
            const long long off = (static_cast<long long>(bh) * p.L1 + row_begin + n * G + g) * p.stat_pitch + jb * 128 + hf * 64;
#pragma unroll 1
            for (int ch = 0; ch < 8; ++ch) {
              uint32_t sv[8], dv[8];
              tmem_ld8(tST + ch * 8, sv);
              tmem_ld8(tDP + ch * 8, dv);
              const uint4 bv = *reinterpret_cast<const uint4*>(brow + ((ch ^ (key & 7)) << 4));
              const uint32_t bw[4] = {bv.x, bv.y, bv.z, bv.w};
              tmem_ld_wait();
#pragma unroll
              for (int e = 0; e < 8; ++e) {
                float b0, b1;
                unpack2<kBf16>(bw[e >> 1], b0, b1);
                const float bq = (e & 1) ? b1 : b0, sq = __uint_as_float(sv[e]);
                float y = fmaf(sq, p.scale * kLog2e, bq * kLog2e);
                if (recs[ch * 8 + e].w & 0xFFFFu) {
                  // x = s*scale + b exactly as the forward pass formed it; (x - max) is then exact
                  // for x near the max whatever its magnitude; y = (x - max)*log2e - log2(sum)
                  const long long o = off + ch * 8 + e;
                  y = fmaf(fmaf(sq, p.scale, bq) + __ldg(p.lse + o), kLog2e, __ldg(p.lse + p.stat_stride + o));
                  dv[e] = __float_as_uint(__uint_as_float(dv[e]) - __ldg(p.delta + o));
                }
                sv[e] = __float_as_uint(y);
              }
              tmem_st8(tST + ch * 8, sv);
              tmem_st8(tDP + ch * 8, dv);
            }
            tmem_st_wait();
            k1_2 = mk2(1.f, 1.f);
            log2e2 = mk2(0.f, 0.f);
            brow = sZero;
          }
          // One pass over the 64 queries in chunks of 8: S^T and dP^T of a chunk are loaded while the previous one is
          // worked on. P^T (input dtype) and dS^T = P^T * (dP^T - delta), with P in float32, replace them in
          // TMEM; dS^T is also summed into the dBias registers and kept for the dQ operand.
          uint32_t dd[32], ds_free = 1;
          {
            uint32_t sv[2][8], dv[2][8], pp[8];
            uint4 bv[2];
            auto load_bias = [&](int ch) { return *reinterpret_cast<const uint4*>(brow + ((ch ^ (key & 7)) << 4)); };
            tmem_ld8(tST, sv[0]);
            tmem_ld8(tDP, dv[0]);
            bv[0] = load_bias(0);
            tmem_ld_wait();
#pragma unroll
            for (int ch = 0; ch < 8; ++ch) {
              if (ch < 7) {
                tmem_ld8(tST + (ch + 1) * 8, sv[(ch + 1) & 1]);
                tmem_ld8(tDP + (ch + 1) * 8, dv[(ch + 1) & 1]);
                // a chunk ahead like them: nothing moves across the wait below, and a load behind it shows its latency
                // (the pass alone, two warps per scheduler: 1 700 -> 1 390 cycles; one: 1 310 -> 910)
                bv[(ch + 1) & 1] = load_bias(ch + 1);
              }
              if (ch == 4 && tt > 0) ds_free = mbar_test_wait(bar(C::B_DQDONE + ((tt - 1) & 1)), ((tt - 1) >> 1) & 1);
              const uint32_t bw[4] = {bv[ch & 1].x, bv[ch & 1].y, bv[ch & 1].z, bv[ch & 1].w};
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                float b0, b1, y0, y1, ds0, ds1;
                unpack2<kBf16>(bw[e], b0, b1);
                un2(fma2(mk2(__uint_as_float(sv[ch & 1][2 * e]), __uint_as_float(sv[ch & 1][2 * e + 1])), k1_2,
                         mul2(mk2(b0, b1), log2e2)),
                    y0, y1);
                const float p0 = fast_exp2(y0), p1 = fast_exp2(y1);
                pp[(ch & 1) * 4 + e] = pack2<kBf16>(p0, p1);
                const f32x2 ds =
                    mul2(mk2(p0, p1), mk2(__uint_as_float(dv[ch & 1][2 * e]), __uint_as_float(dv[ch & 1][2 * e + 1])));
                acc[ch * 4 + e] = add2(acc[ch * 4 + e], ds);
                un2(ds, ds0, ds1);
                dd[ch * 4 + e] = pack2<kBf16>(ds0, ds1);
              }
              if (ch < 7) tmem_ld_wait();
              if (ch == 5) {
                // dS^T row of this key into the M-major staging tile (128-byte swizzle): most of it here, under the
                // exponentials. The tile is free again: the previous dQ MMA has read it.
                if (tt > 0) ok = mbar_finish_wait(ds_free, bar(C::B_DQDONE + ((tt - 1) & 1)), ((tt - 1) >> 1) & 1, w, 0x44);
                if (ok) {
#pragma unroll
                  for (int j = 0; j < 5; ++j)
                    st_shared_v4(my_ds + ((j ^ (key & 7)) << 4), dd[4 * j], dd[4 * j + 1], dd[4 * j + 2], dd[4 * j + 3]);
                }
              }
              // the 8 columns of this chunk have been read: their results go to columns 4 ch .. 4 ch + 3
              if (ch & 1) {
                tmem_st8(tST + (ch >> 1) * 8, pp);
                tmem_st8(tDP + (ch >> 1) * 8, dd + (ch >> 1) * 8);
              }
            }
          }
          if (!ok) break;
#pragma unroll
          for (int j = 5; j < 8; ++j)
            st_shared_v4(my_ds + ((j ^ (key & 7)) << 4), dd[4 * j], dd[4 * j + 1], dd[4 * j + 2], dd[4 * j + 3]);
          q_in = mbar_test_wait(bar(C::B_QDOFULL + 2 * slot + hf), ring_par);
          tmem_st_wait();
          fence_proxy_async_smem();
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(bar(C::B_UFULL + hf));
        }
        if (!ok) break;
        // The sums of this query block as two boxes (128 key rows x 32 queries, 128-byte swizzle): one in the block's
        // half bias stage (this thread's row of it, whose bias values nobody else reads), one in the spare box,
        // whose previous contents left while the block was worked on. With one spare box for both halves those are
        // the other half's; a barrier per half, each waited for once per block, never runs a phase ahead.
        b_in = mbar_test_wait(bar(C::B_BIASFULL + (bs ^ 2)), ((nb + 1) >> 1) & 1);
        const int by = C::NX == 2 ? hf : hf ^ 1;                         // who parked there last
        const int use = (C::NX == 2 || hf == 0) ? nb - 1 : nb;           // in which block
        if (use >= 0) {
          ok = mbar_wait_warp(bar(C::B_BOXFREE + by), use & 1, w, 0x4b);
          if (!ok) break;
        }
#pragma unroll
        for (int box = 0; box < 2; ++box) {
          const uint32_t rowa = (box ? smem_u32(sBox + (hf & (C::NX - 1)) * 16384) : smem_u32(sBias + bs * 16384)) + key * 128;
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            float a0, a1, a2, a3;
            un2(acc[box * 16 + 2 * j], a0, a1);
            un2(acc[box * 16 + 2 * j + 1], a2, a3);
            st_shared_v4(rowa + ((j ^ (key & 7)) << 4), __float_as_uint(a0), __float_as_uint(a1), __float_as_uint(a2),
                         __float_as_uint(a3));
          }
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(C::B_BOX + hf));
      }
    }
  }

  // ---------------------------------------------------------------------- tear-down
  tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag) __nanosleep(20000);
  if (warp == 0) tmem_dealloc(tbase, 512);
}

template <int kD, bool kBf16>
int launch_bwd_t(const BwdArgs& a, int NP, cudaStream_t stream) {
  using C = BwdCfg<kD>;
  static PerDeviceOnce smem_attr;
  auto kern = fta_bwd_kernel<kD, kBf16>;
  if (cudaError_t e = ensure_dynamic_smem(smem_attr, kern, C::SMEM_BYTES)) return static_cast<int>(e);
  BwdParams p;
  p.lse = a.lse;
  p.delta = a.delta;
  p.status = a.status;
  p.H = a.H;
  p.L1 = a.L1;
  p.L2 = a.L2;
  p.NP = NP;
  p.BH = a.B * a.H;
  p.scale = a.sm_scale;
  p.stat_pitch = (a.L2 + 127) / 128 * 128;
  p.stat_stride = static_cast<long long>(a.B) * a.H * a.L1 * p.stat_pitch;
  const int grid = a.B * a.H * NP * ((a.L2 + 127) / 128);
  kern<<<grid, kBwdThreads, C::SMEM_BYTES, stream>>>(a.tmQ, a.tmK, a.tmV, a.tmDO, a.tmBiasT, a.tmDQ, a.tmPlane, a.tmDK,
                                                    a.tmDV, a.tmDQ16, p);
  return static_cast<int>(cudaGetLastError());
}

}  // namespace

int bwd_rows_per_cta(int D) { return D == 32 ? BwdCfg<32>::G : BwdCfg<64>::G; }

// Number of private dBias planes == number of row blocks per (b,h,key block). Chosen so that the
// grid (B*H * L2/128 * NP CTAs, one per SM at a time) fills whole waves of the device with
// chains of nearly equal length, with as few planes as that allows.
int bwd_num_planes(int B, int H, int L1, int L2, int D, int sms) {
  const int G = bwd_rows_per_cta(D);
  const int ngroups = (L1 + G - 1) / G;
  const long long base = static_cast<long long>(B) * H * ((L2 + 127) / 128);
  const int np_max = ngroups < 64 ? ngroups : 64;
  auto efficiency = [&](int np) {
    const long long ctas = base * np;
    const long long waves = (ctas + sms - 1) / sms;
    const int chain = (L1 + np - 1) / np;  // rows of the longest chain
    // time ~ waves * chain ; work ~ base * L1 / sms
    return (static_cast<double>(base) * L1 / sms) / (static_cast<double>(waves) * chain);
  };
  // The planes are updated in place all through the kernel, so their footprint should stay inside
  // the L2 cache. While it does (half of the 126 MB), take the best schedule, and the fewest planes
  // among schedules within 1 % of it; beyond that, the FEWEST planes whose schedule is within 7 % of
  // the best one.
  const long long l2p = (L2 + 127) / 128 * 128;
  const double plane_set_bytes = 4.0 * B * H * static_cast<double>(l2p) * l2p;
  const double budget = 64.0 * 1024 * 1024;
  double best_small = -1.0, best_eff = -1.0;
  for (int np = 1; np <= np_max; ++np) {
    const double e = efficiency(np);
    best_eff = e > best_eff ? e : best_eff;
    if (np * plane_set_bytes <= budget) best_small = e > best_small ? e : best_small;
  }
  if (best_small >= 0.93 * best_eff) {
    for (int np = 1; np <= np_max; ++np)
      if (np * plane_set_bytes <= budget && efficiency(np) >= 0.99 * best_small) return np;
  }
  for (int np = 1; np <= np_max; ++np)
    if (efficiency(np) >= 0.93 * best_eff) return np;
  return 1;
}

int launch_bwd(const BwdArgs& a, cudaStream_t stream) {
  const int NP = a.nplanes;
  if (a.D == 32) return a.bf16 ? launch_bwd_t<32, true>(a, NP, stream) : launch_bwd_t<32, false>(a, NP, stream);
  return a.bf16 ? launch_bwd_t<64, true>(a, NP, stream) : launch_bwd_t<64, false>(a, NP, stream);
}

}  // namespace fta
