// Forward triangle attention for sm_100a, four rows at a time in tiles of 64 keys: O = softmax(sm_scale * q k^T + bias) v
// and the softmax statistics, the work of the reference's `_attn_fwd` (flash_tt_attn.py:128-264). `launch_fwd` says which
// problems come here and which go to the kernel with two warpgroups and tiles of 128 keys.
//
// One CTA owns a 128-query block `jb` of one (b,h) and walks a residue class of the groups of kRows consecutive L1 rows back
// to back. Within a group it walks the key blocks once (outer loop) and, inside, the rows, so that one 128 x 64 bias tile
// staged in shared memory serves a tile of every row:
//
//   warps 0, 2  : tcgen05 issuers, half of the rows each (S = Q K^T into TMEM, O += P V with P read from TMEM)
//   warp 1      : TMA producer  (Q tiles once, K/V ring, bias ring)         warp 3 : idle
//   warps 4-    : kRows softmax warpgroups, one row of the group each; thread = query row
//
// What bounds it: a softmax warp's chain from one tile to the next (S out of TMEM, bias, row max, rescaling of O,
// exponentials, P into TMEM, and back through the issuer), which the other warps of its scheduler have to cover. Four
// warpgroups need tiles of 64 keys, since the logits of a tile live in registers (104 a thread); a thread then has one
// row, and its own O accumulator, instead of two. A ragged L2 is padded to 64 keys instead of 128.
// An issuer needs about 1 300 cycles for a tile's Q K^T and P V beside the softmax warps - not for the MMAs, for its
// own instructions: with one for all four rows it was the bound (L768 forward 850 us; two: 692). A warp for each row
// that also does the row's loads is never waited for, and yet slower (736): the softmax warps are then in step often enough
// to queue for the exp2 unit. Issuing from the softmax warps themselves: 933.
// The bias is loaded two vectors ahead of its use (four: 703).
//
// Measured (two warpgroups with tiles of 128 keys -> this kernel, us, D 32 bf16 unless stated): inference B1 H4 L768 722 ->
// 685, L384 105.6 -> 101.4, B4 H8 L256 263 -> 249, L64 29.5 -> 21.4, B1 H8 L317 fp16 174 -> 139, B1 H16 L1 1024 L2 32 136 -> 72,
// D 64 B1 H8 L320 216 -> 190; with statistics and the residual of O L768 765 -> 699, L384 117.6 -> 105.4, B4 H8 L256 302 ->
// 259, D 64 B1 H8 L320 290 -> 218. Of these the 32-byte stores of O and its residual give 59, 14, 45 and 49 us.
//
// The producer and issuer loops run warp-uniformly (all 32 lanes) and only the TMA / MMA instruction itself is issued by
// one elected lane. The O accumulator is rescaled whenever the row max grew, by the thread that owns the query row, before
// P is handed to the PV MMA.
#include "fta_kernels.h"
#include "schedule.h"
#include "tc05.cuh"

#include <type_traits>

namespace fta {

namespace {

constexpr float kLog2e = 1.4426950408889634f;

template <int kD>
struct QuadCfg {
  static constexpr int G = 4;                         // softmax warpgroups == rows in flight
  static constexpr int KB = 64;                       // keys per tile
  static constexpr int NSTAGE = (kD == 32) ? 12 : 6;  // K/V ring depth (tiles)
  static constexpr int NBIAS = (kD == 32) ? 4 : 3;    // bias ring depth (key blocks)
  // D = 64: the O accumulators leave no columns for P beside S; P replaces S
  static constexpr bool P_OVER_S = kD == 64;
  static constexpr int Q_B = 128 * kD * 2;            // 128 queries of one row
  static constexpr int KV_B = KB * kD * 2;            // a K or V tile
  static constexpr int BIAS_B = 128 * KB * 2;         // 128 queries x 64 keys
  static constexpr int OFF_Q = 0;
  static constexpr int OFF_KV = OFF_Q + G * Q_B;
  static constexpr int OFF_BIAS = OFF_KV + NSTAGE * 2 * KV_B;
  static constexpr int OFF_BAR = OFF_BIAS + NBIAS * BIAS_B;
  // barrier slots
  static constexpr int B_QFULL = 0;
  static constexpr int B_QEMPTY = B_QFULL + G;
  static constexpr int B_KVFULL = B_QEMPTY + G;
  static constexpr int B_KVEMPTY = B_KVFULL + NSTAGE;
  static constexpr int B_BIASFULL = B_KVEMPTY + NSTAGE;
  static constexpr int B_BIASEMPTY = B_BIASFULL + NBIAS;
  static constexpr int B_SFULL = B_BIASEMPTY + NBIAS;  // per warpgroup from here
  static constexpr int B_SFREE = B_SFULL + G;
  static constexpr int B_PFULL = B_SFREE + G;
  static constexpr int B_PVDONE = B_PFULL + G;
  static constexpr int NBAR = B_PVDONE + G;
  static constexpr int SMEM_BYTES = OFF_BAR + NBAR * 8 + 16 + 1024;  // + tmem slot/abort + align slack
  static constexpr uint64_t SWZ = (kD == 32) ? kSwz64 : kSwz128;
  static constexpr uint32_t SBO = 8 * kD * 2;  // bytes between 8-row groups of a tile
  // TMEM columns of warpgroup g
  static constexpr uint32_t TM_S = 0;                        // + 64 g
  static constexpr uint32_t TM_P = P_OVER_S ? 0 : 256;       // + P_STEP g
  static constexpr uint32_t P_STEP = P_OVER_S ? 64 : 32;
  static constexpr uint32_t TM_O = P_OVER_S ? 256 : 384;     // + D g
  static_assert(TM_O + G * kD <= 512, "TMEM budget");
};
// threads of a block: four service warps, kRows softmax warpgroups
constexpr int quad_threads(int rows) { return 128 + 128 * rows; }
// Registers per thread after setmaxnreg with four rows: 4 * 104 + 64 = 4 * 112 + 32 = 5 * 96, the block's allotment at launch. At
// D = 64 the softmax warps spill less with 112 than the service warps lose with 32 (B1 H8 L320 training forward 218 -> 208 us,
// inference 190 -> 181); at D = 32, where 104 nearly suffice, it costs L768 0.6 %. A block of two rows has 168 for every thread.
template <int kD>
constexpr int kRegsSoftmax = kD == 32 ? 104 : 112;
template <int kD>
constexpr int kRegsService = kD == 32 ? 64 : 32;

struct QuadParams {
  void* o;
  void* o_resid;  // optional: the part of O lost in rounding to 16 bits, same layout as O
  float* lse;     // nullptr: no statistics
  Status status;
  int H, L1, L2;
  bool wide;                         // every row of O (and of o_resid) starts at a multiple of 32 bytes
  long long so_b, so_h, so_i, so_j;  // element strides of O (D stride is 1)
  float scale;                       // sm_scale
  int stat_pitch;                    // row pitch of the statistics: L2 rounded up to 128
  long long stat_stride;             // elements between the statistics planes
};

// kRows: rows per group == softmax warpgroups
template <int kD, bool kBf16, int kRows>
__global__ void __launch_bounds__(quad_threads(kRows), 1)
fta_fwd_quad_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
               const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmBias,
               const QuadParams p) {
  using C = QuadCfg<kD>;
  constexpr int G = C::G;
  extern __shared__ uint8_t smem_raw[];
  // 1 KB alignment by an offset from the shared array itself, so that the compiler keeps the
  // shared address space (ld.shared / st.shared instead of generic accesses)
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint8_t* sQ = smem + C::OFF_Q;
  uint8_t* sKV = smem + C::OFF_KV;
  uint8_t* sBias = smem + C::OFF_BIAS;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::OFF_BAR);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + C::NBAR);
  int* abort_flag = reinterpret_cast<int*>(tmem_slot + 1);
  const uint32_t bar0 = smem_u32(bars);
  auto bar = [&](int i) { return bar0 + 8u * static_cast<uint32_t>(i); };

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int jb = blockIdx.x, bh = blockIdx.z;
  const int b = bh / p.H, h = bh % p.H;
  // a ragged last key block is padded by the loads (zeros) and masked by the bias (-inf)
  const int nkb = (p.L2 + C::KB - 1) / C::KB;
  // This CTA walks the row groups blockIdx.y, blockIdx.y + gridDim.y, ... ("units") back to back;
  // loads and MMAs of the next unit start while the softmax warps finish the current one.
  // Every unit processes kRows rows: a short last group is padded with rows past L1, which the TMA
  // loads fill with zeros and the epilogue does not store.
  const int ngroups = (p.L1 + kRows - 1) / kRows;
  const int nunits = (ngroups - static_cast<int>(blockIdx.y) + static_cast<int>(gridDim.y) - 1) /
                     static_cast<int>(gridDim.y);
  auto unit_i0 = [&](int u) { return (static_cast<int>(blockIdx.y) + u * static_cast<int>(gridDim.y)) * kRows; };
  const WaitCtx w{smem_u32(abort_flag), p.status.word};

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int i = 0; i < C::NSTAGE; ++i) {
      mbar_init(bar(C::B_KVFULL + i), 1);
      mbar_init(bar(C::B_KVEMPTY + i), 1);
    }
    for (int i = 0; i < C::NBIAS; ++i) {
      mbar_init(bar(C::B_BIASFULL + i), 1);
      mbar_init(bar(C::B_BIASEMPTY + i), 4 * kRows);  // one arrive per softmax warp
    }
    for (int i = 0; i < G; ++i) {
      mbar_init(bar(C::B_QFULL + i), 1);
      mbar_init(bar(C::B_QEMPTY + i), 1);
      mbar_init(bar(C::B_SFULL + i), 1);
      mbar_init(bar(C::B_SFREE + i), 4);  // one arrive per warp of the warpgroup
      mbar_init(bar(C::B_PFULL + i), 4);
      mbar_init(bar(C::B_PVDONE + i), 1);
    }
    mbar_fence_init();
  }
  if (warp == 0) {
    tmem_alloc(smem_u32(tmem_slot), 512);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tbase = *tmem_slot;
  // everything above overlaps the kernel before (the staging of the bias; 12.3 -> 10.5 us at B1 H4 L64 D32)
  grid_dependency_wait();

  if (warp < 4) {
    if constexpr (kRows == 4) reg_dec<kRegsService<kD>>();
    if (warp == 1) {
      // ---------------------------------------------------------------- TMA producer
      if (elect_one()) {
        tma_prefetch_desc(&tmQ);
        tma_prefetch_desc(&tmK);
        tma_prefetch_desc(&tmV);
        tma_prefetch_desc(&tmBias);
      }
      bool ok = true;
      int s = 0, bs = 0;
      uint32_t kv_par = 1, bias_par = 1;  // of the waits for an empty stage
      for (int u = 0; u < nunits && ok; ++u) {
        const int i0 = unit_i0(u);
        for (int kb = 0; kb < nkb && ok; ++kb) {
          ok = mbar_wait_warp(bar(C::B_BIASEMPTY + bs), bias_par, w, 1);
          if (!ok) break;
          if (elect_one()) {
            mbar_expect_tx(bar(C::B_BIASFULL + bs), C::BIAS_B);
            tma_load_4d(smem_u32(sBias + bs * C::BIAS_B), &tmBias, bar(C::B_BIASFULL + bs), kb * C::KB, jb * 128, h, b);
          }
          __syncwarp();
          if (++bs == C::NBIAS) {
            bs = 0;
            bias_par ^= 1u;
          }
          for (int g = 0; g < kRows; ++g) {
            if (kb == 0) {
              // the Q tile of this row slot is free once the last Q K^T of the previous unit is done
              ok = mbar_wait_warp(bar(C::B_QEMPTY + g), (u & 1) ^ 1, w, 11);
              if (!ok) break;
              if (elect_one()) {
                mbar_expect_tx(bar(C::B_QFULL + g), C::Q_B);
                tma_load_5d(smem_u32(sQ + g * C::Q_B), &tmQ, bar(C::B_QFULL + g), 0, jb * 128, i0 + g, h, b);
              }
              __syncwarp();
            }
            ok = mbar_wait_warp(bar(C::B_KVEMPTY + s), kv_par, w, 2);
            if (!ok) break;
            if (elect_one()) {
              mbar_expect_tx(bar(C::B_KVFULL + s), 2 * C::KV_B);
              tma_load_5d(smem_u32(sKV + s * 2 * C::KV_B), &tmK, bar(C::B_KVFULL + s), 0, kb * C::KB, i0 + g, h, b);
              tma_load_5d(smem_u32(sKV + s * 2 * C::KV_B + C::KV_B), &tmV, bar(C::B_KVFULL + s), 0, kb * C::KB, i0 + g, h, b);
            }
            __syncwarp();
            if (++s == C::NSTAGE) {
              s = 0;
              kv_par ^= 1u;
            }
          }
        }
      }
    } else if (warp == 0 || warp == 2) {
      // ---------------------------------------------------------------- MMA issuer
      // Tiles in the order (unit, key block, row); tile t belongs to warpgroup t % kRows. The Q K^T of a warpgroup's next
      // tile is issued before its P V where S and P have columns of their own (its S tile has long been copied out),
      // behind it where P replaces S (the tensor core works in the order of issue).
      constexpr uint32_t idesc_qk = umma_idesc_f16(kBf16 ? 1 : 0, 128, C::KB, 0, 0);
      constexpr uint32_t idesc_pv = umma_idesc_f16(kBf16 ? 1 : 0, 128, kD, 0, 1);
      // Descriptors as 32-bit low words (address and leading-dimension offset); the high word is a constant.
      constexpr uint32_t HI = (C::SBO >> 4) | (1u << 14) | (static_cast<uint32_t>(C::SWZ) << 29);
      auto mk = [](uint32_t lo) { return (static_cast<uint64_t>(HI) << 32) | lo; };
      constexpr uint32_t LK = 1u << 16, LM = (C::SBO >> 4) << 16;  // K-major: lbo = 16 bytes; M-major: lbo = SBO
      const uint32_t lo_q = (smem_u32(sQ) >> 4) | LK, lo_k = (smem_u32(sKV) >> 4) | LK,
                     lo_v = ((smem_u32(sKV) + C::KV_B) >> 4) | LM;
      constexpr uint32_t Q_STEP = C::Q_B >> 4, STAGE_STEP = 2 * C::KV_B >> 4;
      bool ok = true;
      const int ntiles = nunits * nkb;  // per warpgroup
      // the tile whose Q K^T comes next: its number within the warpgroup, row, unit parity, key block, stage
      constexpr int RPI = kRows / 2;           // rows per issuer
      const int g_lo = (warp >> 1) * RPI;
      int qn = 0, qg = g_lo, qkb = 0, qs = g_lo;
      uint32_t qu = 0, qkv = 0;
      // What it waits for is polled before, together: a poll one has to wait for costs 150 cycles.
      uint32_t q_in = 1, kv_in = 1, s_in = 1;
      auto poll_qk = [&]() {
        if (qkb == 0) q_in = mbar_test_wait(bar(C::B_QFULL + qg), qu);
        kv_in = mbar_test_wait(bar(C::B_KVFULL + qs), qkv);
        if (!C::P_OVER_S && qn > 0) s_in = mbar_test_wait(bar(C::B_SFREE + qg), (qn - 1) & 1);
      };
      auto issue_qk = [&]() -> bool {
        if (qkb == 0 && !mbar_finish_wait(q_in, bar(C::B_QFULL + qg), qu, w, 3)) return false;
        if (!mbar_finish_wait(kv_in, bar(C::B_KVFULL + qs), qkv, w, 4)) return false;
        if (!C::P_OVER_S && qn > 0 && !mbar_finish_wait(s_in, bar(C::B_SFREE + qg), (qn - 1) & 1, w, 9)) return false;
        tc_fence_after_sync();
        if (elect_one()) {
#pragma unroll
          for (int ks = 0; ks < kD / 16; ++ks)
            umma_ss(tbase + C::TM_S + qg * 64, mk(lo_q + qg * Q_STEP) + ks * 2, mk(lo_k + qs * STAGE_STEP) + ks * 2, idesc_qk, ks > 0);
          umma_commit(bar(C::B_SFULL + qg));
          if (qkb == nkb - 1) umma_commit(bar(C::B_QEMPTY + qg));  // last use of this unit's Q tile
        }
        __syncwarp();
        ++qs;
        if (++qg == g_lo + RPI) {
          qg = g_lo;
          qs += kRows - RPI;
          ++qn;
          if (++qkb == nkb) {
            qkb = 0;
            qu ^= 1u;
          }
        }
        if (qs >= C::NSTAGE) {
          qs -= C::NSTAGE;
          qkv ^= 1u;
        }
        return true;
      };
      for (int g = 0; g < RPI && ok && ntiles > 0; ++g) {
        poll_qk();
        ok = issue_qk();
      }
      int s = g_lo, kb = 0;
      for (int n = 0; n < ntiles && ok; ++n) {
        const uint32_t acc0 = kb > 0 ? 1u : 0u;
#pragma unroll 1
        for (int g = g_lo; g < g_lo + RPI && ok; ++g) {
          if (n + 1 < ntiles) poll_qk();
          const uint32_t p_in = mbar_test_wait(bar(C::B_PFULL + g), n & 1);
          if (!C::P_OVER_S && n + 1 < ntiles) {
            ok = issue_qk();  // waits until this warpgroup's tile has been copied out
            if (!ok) break;
          }
          ok = mbar_finish_wait(p_in, bar(C::B_PFULL + g), n & 1, w, 5);
          if (!ok) break;
          tc_fence_after_sync();
          if (elect_one()) {
#pragma unroll
            for (int ks = 0; ks < C::KB / 16; ++ks)
              umma_ts(tbase + C::TM_O + g * kD, tbase + C::TM_P + g * C::P_STEP + ks * 8,
                      mk(lo_v + s * STAGE_STEP) + ks * ((2 * C::SBO) >> 4), idesc_pv, ks > 0 ? 1u : acc0);
            umma_commit(bar(C::B_PVDONE + g));
            umma_commit(bar(C::B_KVEMPTY + s));
          }
          __syncwarp();
          if (++s >= C::NSTAGE) s -= C::NSTAGE;
          if (C::P_OVER_S && n + 1 < ntiles) ok = issue_qk();
        }
        s += kRows - RPI;
        if (s >= C::NSTAGE) s -= C::NSTAGE;
        if (++kb == nkb) kb = 0;
      }
    }
  } else {
    // ------------------------------------------------------------------ softmax warpgroups
    if constexpr (kRows == 4) reg_inc<kRegsSoftmax<kD>>();
    const int g = (warp >> 2) - 1;           // warpgroup == row of the group
    const int row = (warp & 3) * 32 + lane;  // query row of the tile == TMEM lane
    const uint32_t lane_off = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t tS = tbase + C::TM_S + g * 64 + lane_off;
    const uint32_t tP = tbase + C::TM_P + g * C::P_STEP + lane_off;
    const uint32_t tO = tbase + C::TM_O + g * kD + lane_off;
    const f32x2 scale2 = mk2(p.scale, p.scale);
    const f32x2 log2e2 = mk2(kLog2e, kLog2e);
    int n = 0, bs = 0;
    uint32_t bias_par = 0, s_in = 0, b_in = 0;
    bool ok = true;
    for (int u = 0; u < nunits && ok; ++u) {
      float m_used = -INFINITY, l_run = 0.f;  // running max (natural-log units) and running sum
#pragma unroll 1
      for (int kb = 0; kb < nkb; ++kb, ++n) {
        const uint8_t* brow = sBias + bs * C::BIAS_B + row * 128;
        ok = mbar_finish_wait(b_in, bar(C::B_BIASFULL + bs), bias_par, w, 7);
        if (!ok) break;
        constexpr int kAhead = kRows == 4 ? 2 : 7;  // vectors of the bias loaded before S; with four rows no register is left for more
        uint4 bv[8];
#pragma unroll
        for (int c = 0; c < kAhead; ++c) bv[c] = *reinterpret_cast<const uint4*>(brow + ((c ^ (row & 7)) << 4));
        ok = mbar_finish_wait(s_in, bar(C::B_SFULL + g), n & 1, w, 6);
        if (!ok) break;
        tc_fence_after_sync();
        uint32_t sr[64];
        tmem_ld32(tS, sr);
        tmem_ld32(tS + 32, sr + 32);
        tmem_ld_wait();
        if constexpr (!C::P_OVER_S) {
          // the S columns may now be overwritten by the next Q K^T of this warpgroup
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(bar(C::B_SFREE + g));
        }
        // this row's previous P V: the P columns are free and O may be rescaled once it is done
        uint32_t pv_in = 1;
        if (n > 0) pv_in = mbar_test_wait(bar(C::B_PVDONE + g), (n - 1) & 1);
        // pass 1: x = s*scale + bias (natural-log units), row max
        float mx0 = -INFINITY, mx1 = -INFINITY, mx2 = -INFINITY, mx3 = -INFINITY;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          if (c < 8 - kAhead) bv[c + kAhead] = *reinterpret_cast<const uint4*>(brow + (((c + kAhead) ^ (row & 7)) << 4));
          const uint32_t bw[4] = {bv[c].x, bv[c].y, bv[c].z, bv[c].w};
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            float b0, b1, x0, x1;
            unpack2<kBf16>(bw[e], b0, b1);
            const f32x2 x = fma2(mk2(__uint_as_float(sr[c * 8 + 2 * e]), __uint_as_float(sr[c * 8 + 2 * e + 1])),
                                 scale2, mk2(b0, b1));
            un2(x, x0, x1);
            sr[c * 8 + 2 * e] = __float_as_uint(x0);
            sr[c * 8 + 2 * e + 1] = __float_as_uint(x1);
            if (e == 0) mx0 = max3(mx0, x0, x1);
            else if (e == 1) mx1 = max3(mx1, x0, x1);
            else if (e == 2) mx2 = max3(mx2, x0, x1);
            else mx3 = max3(mx3, x0, x1);
          }
        }
        const float mx = fmaxf(fmaxf(mx0, mx1), fmaxf(mx2, mx3));
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(C::B_BIASEMPTY + bs));
        if (++bs == C::NBIAS) {
          bs = 0;
          bias_par ^= 1u;
        }
        // The reference maximum follows the running row maximum exactly (the O accumulator is rescaled
        // whenever it grows), so the largest probabilities of a row are powers of two times an exactly
        // representable value when they are rounded to 16 bits for the PV MMA. Letting the reference
        // lag (rescaling only after a growth of 2^8) costs the same time here and doubles the error
        // of O and of delta = rowsum(dO * O) on peaked rows, which dBias then sums over all L1 rows.
        const bool need = mx > m_used;
        const float m_new = need ? mx : m_used;
        const float m_safe = (m_new == -INFINITY) ? 0.f : m_new;
        const float alpha = need ? fast_exp2((m_used - m_safe) * kLog2e) : 1.0f;
        m_used = m_new;
        if (n > 0) {
          ok = mbar_finish_wait(pv_in, bar(C::B_PVDONE + g), (n - 1) & 1, w, 10);
          if (!ok) break;
        }
        if (kb > 0 && __any_sync(0xffffffffu, need)) {
          tc_fence_after_sync();
          const f32x2 alpha2 = mk2(alpha, alpha);
#pragma unroll
          for (int c = 0; c < kD / 16; ++c) {
            uint32_t orr[16];
            tmem_ld16(tO + c * 16, orr);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              float o0, o1;
              un2(mul2(mk2(__uint_as_float(orr[2 * j]), __uint_as_float(orr[2 * j + 1])), alpha2), o0, o1);
              orr[2 * j] = __float_as_uint(o0);
              orr[2 * j + 1] = __float_as_uint(o1);
            }
            tmem_st16(tO + c * 16, orr);
          }
        }
        // pass 2: p = 2^((x - m) * log2e), row sum, pack, hand P to the tensor core through TMEM
        // One fused multiply-add per pair while every row max of the warp is moderate; rows with a
        // huge |max| (keys masked with -1e9) need (x - m) formed first: it is exact when x is close
        // to m whatever their magnitude, whereas x*log2e - m*log2e would round m*log2e to the ulp
        // of 1e9.
        f32x2 sum2a = mk2(0.f, 0.f), sum2b = mk2(0.f, 0.f);
        const bool moderate = __all_sync(0xffffffffu, fabsf(m_safe) <= 1.0e4f);
        if (!moderate) {
          const f32x2 nm2 = mk2(-m_safe, -m_safe);
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            float x0, x1;
            un2(add2(mk2(__uint_as_float(sr[2 * j]), __uint_as_float(sr[2 * j + 1])), nm2), x0, x1);
            sr[2 * j] = __float_as_uint(x0);
            sr[2 * j + 1] = __float_as_uint(x1);
          }
        }
        const float nml = moderate ? -m_safe * kLog2e : 0.f;
        const f32x2 nml2 = mk2(nml, nml);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint32_t pk[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            float y0, y1;
            un2(fma2(mk2(__uint_as_float(sr[c * 16 + 2 * j]), __uint_as_float(sr[c * 16 + 2 * j + 1])), log2e2, nml2), y0, y1);
            const float p0 = fast_exp2(y0), p1 = fast_exp2(y1);
            if (j & 1) sum2b = add2(sum2b, mk2(p0, p1));
            else sum2a = add2(sum2a, mk2(p0, p1));
            pk[j] = pack2<kBf16>(p0, p1);
          }
          tmem_st8(tP + c * 8, pk);
        }
        float s0, s1;
        un2(add2(sum2a, sum2b), s0, s1);
        s_in = mbar_test_wait(bar(C::B_SFULL + g), (n + 1) & 1);  // of the next tile
        b_in = mbar_test_wait(bar(C::B_BIASFULL + bs), bias_par);
        tmem_st_wait();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(C::B_PFULL + g));
        l_run = l_run * alpha + (s0 + s1);
      }
      if (!ok) break;

      // epilogue of the row: wait for the last PV, normalise, store O and the log-sum-exp
      ok = mbar_wait_warp(bar(C::B_PVDONE + g), (n - 1) & 1, w, 8);
      if (!ok) break;
      tc_fence_after_sync();
      const int i = unit_i0(u) + g;
      const float m_safe = (m_used == -INFINITY) ? 0.f : m_used;
      // a row whose every key is masked has an empty sum: O = 0 and statistics that make the
      // backward pass recompute P = 0
      const float inv = l_run > 0.f ? 1.0f / l_run : 0.f;
      const int j = jb * 128 + row;
      const bool live = i < p.L1 && j < p.L2;  // padding rows of a short group / a ragged query block
      const long long ooff = b * p.so_b + h * p.so_h + static_cast<long long>(i) * p.so_i +
                             static_cast<long long>(j) * p.so_j;
      uint16_t* optr = reinterpret_cast<uint16_t*>(p.o) + ooff;
      // O - dtype(O), rounded to the same dtype: with it the backward preprocess forms
      // delta = rowsum(dO * O) from O to 16 mantissa bits instead of 8 (bf16)
      uint16_t* rptr = p.o_resid ? reinterpret_cast<uint16_t*>(p.o_resid) + ooff : nullptr;
#pragma unroll
      for (int c = 0; c < kD / 32; ++c) {
        uint32_t orr[32];
        tmem_ld32(tO + c * 32, orr);
        tmem_ld_wait();
        if (live) {
#pragma unroll
          for (int v = 0; v < 2; ++v) {
            uint32_t ow[8], rw[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              const float o0 = __uint_as_float(orr[v * 16 + 2 * e]) * inv, o1 = __uint_as_float(orr[v * 16 + 2 * e + 1]) * inv;
              float r0, r1;
              ow[e] = pack2<kBf16>(o0, o1);
              unpack2<kBf16>(ow[e], r0, r1);
              rw[e] = pack2<kBf16>(o0 - r0, o1 - r1);
            }
            if (p.wide) {
              st_global_v8(optr + c * 32 + v * 16, ow);
              if (rptr) st_global_v8(rptr + c * 32 + v * 16, rw);
            } else {
              uint4* o4 = reinterpret_cast<uint4*>(optr + c * 32 + v * 16);
              o4[0] = make_uint4(ow[0], ow[1], ow[2], ow[3]);
              o4[1] = make_uint4(ow[4], ow[5], ow[6], ow[7]);
              if (rptr) {
                uint4* r4 = reinterpret_cast<uint4*>(rptr + c * 32 + v * 16);
                r4[0] = make_uint4(rw[0], rw[1], rw[2], rw[3]);
                r4[1] = make_uint4(rw[4], rw[5], rw[6], rw[7]);
              }
            }
          }
        }
      }
      if (i < p.L1 && p.lse != nullptr) {
        float m_safe_out = m_safe;
        // softmax statistics for the backward pass: -max (natural-log units) and -log2(sum).
        // Kept apart: their sum in one float would lose log2(sum) when |max| is huge.
        // (queries past L2 in a ragged block get 0 / -inf / -inf: whatever their logits, P = 0)
        const long long ridx = (static_cast<long long>(bh) * p.L1 + i) * p.stat_pitch + j;
        const bool empty = !(l_run > 0.f) || j >= p.L2;
        const float nl = empty ? -INFINITY : -log2f(l_run);
        if (j >= p.L2) m_safe_out = 0.f;
        p.lse[ridx] = -m_safe_out;
        p.lse[p.stat_stride + ridx] = nl;
        // plane 2: both in one number, c = -(max*log2e + log2 sum), for rows where that loses
        // nothing; NaN marks rows whose max is so large (fully masked rows) that the
        // backward pass must use the two parts separately
        p.lse[2 * p.stat_stride + ridx] =
            (fabsf(m_safe_out) > 1.0e4f) ? __int_as_float(0x7fc00000) : fmaf(-m_safe_out, kLog2e, nl);
      }
    }
  }

  // ---------------------------------------------------------------------- tear-down
  tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag) __nanosleep(20000);  // let copies already in flight land before the CTA exits
  if (threadIdx.x == 0 && (*abort_flag || (blockIdx.x | blockIdx.y | blockIdx.z) == 0))
    publish_status(p.status.word, p.status.mirror);
  if (warp == 0) tmem_dealloc(tbase, 512);
}

template <int kD, bool kBf16, int kRows>
int launch_quad_t(const FwdArgs& a, cudaStream_t stream) {
  using C = QuadCfg<kD>;
  static_assert(kRows <= C::G);
  static PerDeviceOnce smem_attr;
  auto kern = fta_fwd_quad_kernel<kD, kBf16, kRows>;
  if (cudaError_t e = ensure_dynamic_smem(smem_attr, kern, C::SMEM_BYTES)) return static_cast<int>(e);
  QuadParams p;
  p.o = a.o;
  p.o_resid = a.o_resid;
  p.lse = a.lse;
  p.status = a.status;
  p.H = a.H;
  p.L1 = a.L1;
  p.L2 = a.L2;
  // whole 32-byte sectors per store: 16 bytes at a time, 64 or 128 apart from lane to lane, each sector leaves the SM twice
  p.wide = (reinterpret_cast<uintptr_t>(a.o) | reinterpret_cast<uintptr_t>(a.o_resid)) % 32 == 0 && a.so[0] % 16 == 0 &&
           a.so[1] % 16 == 0 && a.so[2] % 16 == 0 && a.so[3] % 16 == 0;
  p.so_b = a.so[0];
  p.so_h = a.so[1];
  p.so_i = a.so[2];
  p.so_j = a.so[3];
  p.scale = a.sm_scale;
  p.stat_pitch = (a.L2 + 127) / 128 * 128;
  p.stat_stride = static_cast<long long>(a.B) * a.H * a.L1 * p.stat_pitch;
  const long long per = static_cast<long long>((a.L2 + 127) / 128) * a.B * a.H;
  const int grid_y = fwd_grid_rows((a.L1 + kRows - 1) / kRows, per, num_sms());
  dim3 grid((a.L2 + 127) / 128, grid_y, a.B * a.H);
  return static_cast<int>(launch_overlapped(kern, grid, quad_threads(kRows), C::SMEM_BYTES, stream, a.tmQ, a.tmK, a.tmV, a.tmBias, p));
}

}  // namespace

int launch_fwd_quad(const FwdArgs& a, cudaStream_t stream) {
  // A problem that leaves SMs idle is bound by the chain of one CTA: groups of two rows halve it, as long as they all fit in
  // one wave. The rows are a template argument: as a run-time value they cost the long problems 4 %.
  const bool two_rows = static_cast<long long>((a.L2 + 127) / 128) * a.B * a.H * ((a.L1 + 1) / 2) <= num_sms();
  auto go = [&](auto d) {
    constexpr int D = decltype(d)::value;
    if (two_rows) return a.bf16 ? launch_quad_t<D, true, 2>(a, stream) : launch_quad_t<D, false, 2>(a, stream);
    return a.bf16 ? launch_quad_t<D, true, 4>(a, stream) : launch_quad_t<D, false, 4>(a, stream);
  };
  return a.D == 32 ? go(std::integral_constant<int, 32>{}) : go(std::integral_constant<int, 64>{});
}

}  // namespace fta
