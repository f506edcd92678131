// Causal grouped-query flash attention, backward, with P and dS kept in tensor memory.
//
// Same three-kernel split and the same contract as attention_bwd.cu (delta, dK/dV, dQ); what changes
// is where the softmax threads put their results.  There P and dS go to shared memory as swizzled bf16
// tiles, which costs a shared-memory write pass, an async-proxy fence and a serialising "buffer free"
// handshake per operand.  Here they are written with tcgen05.st over the fp32 values they were
// computed from and consumed by the gradient MMAs as the A operand FROM tensor memory:
//
//   attn_dq_tmem_kernel     work items (query tile, head).  S = Q K_j^T alternates between two score
//                           regions, dP = dO V_j^T has one.  The softmax threads pull both into
//                           registers (all loads in flight, one wait), report that (the dP region is
//                           then free for tile j+1), form dS = P (dP - delta) and store it, packed,
//                           into the score region they read S from.  dQ += dS K_j takes A = dS from
//                           tensor memory.  The MMAs of tile j+1 run under the softmax of tile j.
//   attn_dkdv_tmem_kernel   one CTA per (key tile, kv head), transposed: S^T = K Q_i^T and
//                           dP^T = V dO_i^T put the KEY rows on the tensor-memory lanes, so P^T and
//                           dS^T come out in the layout that dV += P^T dO_i and dK += dS^T Q_i need as
//                           A operands.  The row statistics (log-sum-exp and delta) are then per
//                           COLUMN; every item's 2 x 128 values are staged in shared memory.
//
// A thread overwrites only tensor-memory columns it has read itself, so no thread can clobber a value
// another warp still needs.  Waits are bounded as everywhere (common.cuh).
#include "attention_common.cuh"

namespace tft {
namespace attn {

// dS (or P) of 32 score columns as 16 packed bf16 pairs.
__device__ __forceinline__ void pack32(const float (&v)[32], uint32_t (&out)[16]) {
#pragma unroll
  for (int i = 0; i < 16; ++i) out[i] = pack_bf16(v[2 * i], v[2 * i + 1]);
}

// Tensor-memory column of k-step `k` (16 contraction indices = 8 packed columns) of an A operand that
// the two threads of a row wrote into the first 32 columns of their own 64-column halves.
__device__ __forceinline__ uint32_t packed_kstep(uint32_t region, int k) {
  return region + (k < 4 ? k * 8 : 64 + (k - 4) * 8);
}

// ------------------------------------------------------------------ dQ
// Persistent: one CTA per SM walks over (query tile, head, batch) work items, heaviest first and in alternating direction
// from round to round, which evens out the triangular lengths.  Loads of the next item's Q and dO start when the last
// products that read the present ones have run, so they travel under the last softmax and the store of dQ.  With one
// item per CTA (seven CTAs per SM at S 4096, 32 heads) launch, tensor-memory allocation, first loads and store cost 10.7
// thousand cycles an item, a fifth of the time.  S 4096, 32/8 heads of 128: 156 us for 164; two of 2048, heads of 64: 69 for 82.
// At head dimension 64 the softmax threads set the pace (1024 cycles of MUFU a tile against 768 of products), so two groups
// of eight warps take turns on the key tiles, and Q, dO and the accumulator have two buffers: one group stores an item's
// dQ while the other works on the next item.
template <int HD>
struct DqTmemSmem {
  static constexpr int KSTAGES = 3, VSTAGES = 2;
  static constexpr int NG = HD == 64 ? 2 : 1;  // groups of 8 softmax warps
  static constexpr int QB = HD == 64 ? 2 : 1;  // buffers of Q, dO and dQ
  static constexpr int THREADS = 64 + NG * 256;
  static constexpr uint32_t TILE = BLK * HD * 2;
  static constexpr uint32_t Q = 0, DO = QB * TILE, K = 2 * QB * TILE, V = K + KSTAGES * TILE;
  static constexpr uint32_t BARS = V + VSTAGES * TILE;
  static constexpr uint32_t TOTAL = BARS + 256 + 1024;
};
enum DqTmemBar {
  TQ_QDO_FULL0 = 0, TQ_QDO_EMPTY0 = 2, TQ_K_FULL0 = 4, TQ_K_EMPTY0 = 7, TQ_V_FULL0 = 10, TQ_V_EMPTY0 = 12,
  // by parity of the tile's number in this CTA: inputs complete / read into registers / dS stored
  TQ_SDP_FULL0 = 14, TQ_LOADED0 = 16, TQ_DS_READY0 = 18,
  TQ_DQ_EMPTY0 = 20, TQ_DQ_FULL0 = 22, NUM_TQ_BARS = 24
};
static_assert(8 * NUM_TQ_BARS + 16 <= 256, "barriers, tensor-memory address and abort flag share 256 bytes");

struct DqItem {
  int qt, head, batch;
};
// Item of round i for this CTA; -1 as query tile if there is none.
__device__ __forceinline__ DqItem dq_item(int i, int n_tiles, int Hq, int B) {
  const int G = gridDim.x, per_tile = Hq * B;
  const int w = i * G + ((i & 1) ? G - 1 - static_cast<int>(blockIdx.x) : static_cast<int>(blockIdx.x));
  DqItem it;
  it.qt = w < n_tiles * per_tile ? n_tiles - 1 - w / per_tile : -1;
  const int rest = w % per_tile;
  it.head = rest % Hq;
  it.batch = rest / Hq;
  return it;
}

template <int HD>
__global__ void __launch_bounds__(DqTmemSmem<HD>::THREADS, 1)
attn_dq_tmem_kernel(const __grid_constant__ CUtensorMap tq, const __grid_constant__ CUtensorMap tk,
                    const __grid_constant__ CUtensorMap tv, const __grid_constant__ CUtensorMap tdo,
                    const float* __restrict__ LSE, const float* __restrict__ delta, __nv_bfloat16* __restrict__ dQ,
                    int B, int S, int Hq, int Hkv, long long lddq, float scale, float scale_log2, int* status) {
  using L = DqTmemSmem<HD>;
  constexpr int KS = L::KSTAGES, VS = L::VSTAGES, NG = L::NG, QB = L::QB;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t* smem = smem_raw + (base - raw);
  const uint32_t bar0 = base + L::BARS;
  auto bar = [&](int i) { return bar0 + 8u * i; };
  volatile uint32_t* tmem_holder = reinterpret_cast<volatile uint32_t*>(smem + L::BARS + 8 * NUM_TQ_BARS);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + L::BARS + 8 * NUM_TQ_BARS + 8);

  const int warp = uniform_warp_index(), lane = threadIdx.x & 31;
  const int n_tiles = (S + BLK - 1) / BLK;
  const int group = Hq / Hkv;
  const int rounds = (n_tiles * Hq * B + gridDim.x - 1) / gridDim.x;

  if (threadIdx.x == 0) {
    for (int i = 0; i < NUM_TQ_BARS; ++i) mbar_init(bar(i), (i >= TQ_LOADED0 && i < TQ_DQ_FULL0) ? 8 : 1);  // one arrival per warp of a group
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tq);
    tma_prefetch_desc(&tk);
    tma_prefetch_desc(&tv);
    tma_prefetch_desc(&tdo);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_holder)), 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_holder;
  auto t_s = [&](int c) { return tmem_base + static_cast<uint32_t>(c & 1) * 128u; };  // scores, later dS, of tile c
  const uint32_t t_dp = tmem_base + 256;
  auto t_dq = [&](int u) { return tmem_base + 384u + static_cast<uint32_t>(u % QB) * HD; };
  // u counts the items of this CTA, c its key tiles; both run on from item to item, and with them every barrier phase

  if (warp == 0) {
    if (lane == 0) {
      bool ok = true;
      for (int i = 0, u = 0, c = 0; i < rounds && ok; ++i) {
        const DqItem w = dq_item(i, n_tiles, Hq, B);
        if (w.qt < 0) continue;
        const int qb = u % QB, kv_head = w.head / group;
        if (!mbar_wait(bar(TQ_QDO_EMPTY0 + qb), ((u / QB) & 1) ^ 1, abort_flag)) break;
        mbar_expect_tx(bar(TQ_QDO_FULL0 + qb), 2 * L::TILE);
        load_tile<HD>(base + L::Q + qb * L::TILE, &tq, bar(TQ_QDO_FULL0 + qb), w.head, w.qt * BLK, w.batch);
        load_tile<HD>(base + L::DO + qb * L::TILE, &tdo, bar(TQ_QDO_FULL0 + qb), w.head, w.qt * BLK, w.batch);
        for (int j = 0; j <= w.qt; ++j, ++c) {
          const int ks = c % KS, vs = c % VS;
          ok = mbar_wait(bar(TQ_K_EMPTY0 + ks), ((c / KS) & 1) ^ 1, abort_flag);
          if (!ok) break;
          mbar_expect_tx(bar(TQ_K_FULL0 + ks), L::TILE);
          load_tile<HD>(base + L::K + ks * L::TILE, &tk, bar(TQ_K_FULL0 + ks), kv_head, j * BLK, w.batch);
          ok = mbar_wait(bar(TQ_V_EMPTY0 + vs), ((c / VS) & 1) ^ 1, abort_flag);
          if (!ok) break;
          mbar_expect_tx(bar(TQ_V_FULL0 + vs), L::TILE);
          load_tile<HD>(base + L::V + vs * L::TILE, &tv, bar(TQ_V_FULL0 + vs), kv_head, j * BLK, w.batch);
        }
        ++u;
      }
    }
  } else if (warp == 1) {
    const uint32_t leader = elect_one();
    constexpr uint32_t idesc_s = make_idesc_bf16(BLK, BLK, false, false);
    constexpr uint32_t idesc_q = make_idesc_bf16(BLK, HD, false, true);
    auto issue_s = [&](int c, uint32_t sq) -> bool {  // S(c) = Q K^T into the score region of tile c
      const int ks = c % KS;
      if (!mbar_wait_warp(bar(TQ_K_FULL0 + ks), (c / KS) & 1, abort_flag)) return false;
      tc_fence_after();
#pragma unroll
      for (int k = 0; k < HD / 16; ++k)
        umma_bf16_elect(leader, t_s(c), kmajor_desc(sq, k), kmajor_desc(base + L::K + ks * L::TILE, k), idesc_s, k != 0);
      return true;
    };
    // dP(c) = dO V^T, once the softmax threads hold dP(c - 1) in registers; with it the inputs of softmax(c) are complete
    auto issue_dp = [&](int c, uint32_t sdo) -> bool {
      const int vs = c % VS;
      if (c > 0 && !mbar_wait_warp(bar(TQ_LOADED0 + ((c - 1) & 1)), ((c - 1) >> 1) & 1, abort_flag)) return false;
      if (!mbar_wait_warp(bar(TQ_V_FULL0 + vs), (c / VS) & 1, abort_flag)) return false;
      tc_fence_after();
#pragma unroll
      for (int k = 0; k < HD / 16; ++k)
        umma_bf16_elect(leader, t_dp, kmajor_desc(sdo, k), kmajor_desc(base + L::V + vs * L::TILE, k), idesc_s, k != 0);
      umma_commit_elect(leader, bar(TQ_SDP_FULL0 + (c & 1)));
      umma_commit_elect(leader, bar(TQ_V_EMPTY0 + vs));
      return true;
    };
    bool ok = true;
    for (int i = 0, u = 0, c0 = 0; i < rounds && ok; ++i) {
      const DqItem w = dq_item(i, n_tiles, Hq, B);
      if (w.qt < 0) continue;
      const int qb = u % QB, n_kv = w.qt + 1;
      const uint32_t sq = base + L::Q + qb * L::TILE, sdo = base + L::DO + qb * L::TILE, par = (u / QB) & 1;
      ok = mbar_wait_warp(bar(TQ_QDO_FULL0 + qb), par, abort_flag) && issue_s(c0, sq) && issue_dp(c0, sdo);
      if (ok && n_kv > 1) ok = issue_s(c0 + 1, sq);
      if (ok && n_kv == 1) umma_commit_elect(leader, bar(TQ_QDO_EMPTY0 + qb));
      for (int j = 0; j < n_kv && ok; ++j) {
        const int c = c0 + j;
        if (j + 1 < n_kv) {
          if (!issue_dp(c + 1, sdo)) { ok = false; break; }
          if (j + 2 == n_kv) umma_commit_elect(leader, bar(TQ_QDO_EMPTY0 + qb));  // nothing reads this Q and dO any more
        }
        if (!mbar_wait_warp(bar(TQ_DS_READY0 + (c & 1)), (c >> 1) & 1, abort_flag)) { ok = false; break; }
        if (j == 0 && !mbar_wait_warp(bar(TQ_DQ_EMPTY0 + qb), par ^ 1, abort_flag)) { ok = false; break; }
        tc_fence_after();
        // dQ += dS K_j   (contraction over the 128 key rows; A = dS from tensor memory)
        const uint32_t sk = base + L::K + (c % KS) * L::TILE;
#pragma unroll
        for (int k = 0; k < BLK / 16; ++k)
          umma_bf16_ts_elect(leader, t_dq(u), packed_kstep(t_s(c), k), mnmajor_desc(sk, k), idesc_q, (j | k) != 0);
        umma_commit_elect(leader, bar(TQ_K_EMPTY0 + (c % KS)));
        // the score region of tile c is free again once those MMAs have run (in order): tile c + 2 goes there
        if (j + 2 < n_kv && !issue_s(c + 2, sq)) { ok = false; break; }
      }
      if (ok) umma_commit_elect(leader, bar(TQ_DQ_FULL0 + qb));
      c0 += n_kv;
      ++u;
    }
  } else {
    const int q = warp & 3;
    const int g = (warp - 2) >> 3;           // group: takes the tiles c with c % NG == g
    const int half = ((warp - 2) >> 2) & 1;  // two threads per row: key columns [0,64) and [64,128)
    const int r = q * 32 + lane;
    const uint32_t lane_addr = static_cast<uint32_t>(q * 32) << 16;
    bool ok = true;
    for (int i = 0, u = 0, c0 = 0; i < rounds && ok; ++i) {
      const DqItem w = dq_item(i, n_tiles, Hq, B);
      if (w.qt < 0) continue;
      const int row = w.qt * BLK + r, n_kv = w.qt + 1;
      const long long stat = (static_cast<long long>(w.batch) * Hq + w.head) * S + row;
      const float lse = row < S ? LSE[stat] : 0.f;
      const float dl = row < S ? delta[stat] : 0.f;
      for (int j = NG == 1 ? 0 : (c0 + g) & 1; j < n_kv; j += NG) {
        const int c = c0 + j;
        if (!mbar_wait_warp(bar(TQ_SDP_FULL0 + (c & 1)), (c >> 1) & 1, abort_flag)) { ok = false; break; }
        tc_fence_after();
        const bool diag = (j == w.qt);
        const uint32_t my_s = t_s(c) + lane_addr + half * 64, my_dp = t_dp + lane_addr + half * 64;
        auto loaded = [&]() {
          tmem_ld_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(bar(TQ_LOADED0 + (c & 1)));
        };
        uint32_t sv[2][32], dv[2][32];
        if (NG == 1) {  // everything in flight at once; two groups have fewer registers each and work under one another's waits
#pragma unroll
          for (int cc = 0; cc < 2; ++cc) {
            tmem_ld_32x32(my_s + cc * 32, sv[cc]);
            tmem_ld_32x32(my_dp + cc * 32, dv[cc]);
          }
          loaded();
        }
#pragma unroll
        for (int cc = 0; cc < 2; ++cc) {
          if (NG == 2) {
            tmem_ld_32x32(my_s + cc * 32, sv[cc]);
            tmem_ld_32x32(my_dp + cc * 32, dv[cc]);
            if (cc == 0)
              tmem_ld_wait();
            else
              loaded();
          }
          const int col0 = half * 64 + cc * 32;
          float ds[32];
          if (diag) {  // rows beyond the sequence need no mask: a row of dS reaches its own row of dQ only
#pragma unroll
            for (int i2 = 0; i2 < 32; ++i2) {
              const bool keep = (col0 + i2) <= r;
              const float p = keep ? fast_exp2(__uint_as_float(sv[cc][i2]) * scale_log2 - lse) : 0.f;
              ds[i2] = p * (__uint_as_float(dv[cc][i2]) - dl);
            }
          } else {
#pragma unroll
            for (int i2 = 0; i2 < 32; ++i2) {
              const float p = fast_exp2(__uint_as_float(sv[cc][i2]) * scale_log2 - lse);
              ds[i2] = p * (__uint_as_float(dv[cc][i2]) - dl);
            }
          }
          uint32_t packed[16];
          pack32(ds, packed);
          tmem_st_32x16(my_s + cc * 16, packed);  // over score columns this thread has already read
        }
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();  // the lanes' stores are ordered before the one arrival of the warp
        if (lane == 0) mbar_arrive(bar(TQ_DS_READY0 + (c & 1)));
      }
      c0 += n_kv;
      if (ok && (c0 - 1) % NG == g) {  // the group of the last tile stores the item
        const int qb = u % QB;
        ok = mbar_wait_warp(bar(TQ_DQ_FULL0 + qb), (u / QB) & 1, abort_flag);
        if (ok) {
          tc_fence_after();
          const long long tok = static_cast<long long>(w.batch) * S + row;
          store_acc<HD / 2>(t_dq(u) + lane_addr + half * (HD / 2), dQ + tok * lddq + w.head * HD + half * (HD / 2), lddq, scale, S - row);
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(bar(TQ_DQ_EMPTY0 + qb));
        }
      }
      ++u;
    }
    tc_fence_before();
  }

  __syncthreads();
  if (*abort_flag) {
    const long long t0 = clock64();
    while (clock64() - t0 < 2000000LL) { }
    if (threadIdx.x == 0 && status) atomicCAS(status, 0, static_cast<int>(kTimeoutBarrier));
  }
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

template <int HD>
int launch_dq_tmem(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& tdo,
                   const float* lse, const float* delta, void* dq, int B, int S, int Hq, int Hkv, long long lddq,
                   float scale, int* status, cudaStream_t stream) {
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(attn_dq_tmem_kernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         DqTmemSmem<HD>::TOTAL);
    if (e != cudaSuccess) return static_cast<int>(e);
    configured = true;
  }
  const int items = (S + BLK - 1) / BLK * Hq * B, sms = sm_count();
  attn_dq_tmem_kernel<HD><<<items < sms ? items : sms, DqTmemSmem<HD>::THREADS, DqTmemSmem<HD>::TOTAL, stream>>>(
      tq, tk, tv, tdo, lse, delta, static_cast<__nv_bfloat16*>(dq), B, S, Hq, Hkv, lddq, scale,
      scale * 1.4426950408889634f, status);
  return static_cast<int>(cudaGetLastError());
}

// ------------------------------------------------------------------ dK, dV (transposed scores), head dimension 128
// An item is one query head of the group x one query tile.  Tensor-core order per item t:
//
//   dV(t) queries 0-63 | dV(t) 64-127 | S(t+1) | dK(t) 0-63 | dK(t) 64-127 | dP(t+1)
//
// The softmax threads work on the first 64 query columns of an item before the last 64 and announce the two halves
// separately, so the gradient products start under the second half of the exponentials.  S(t+1) follows dV(t) directly and
// runs under the formation of dS(t); dP(t+1) comes last, where nobody waits for it.  The two accumulators take half of the
// tensor memory, which leaves one score region.
// What bounds it: the exponentials of an item take 1024 cycles of the MUFU unit (16 a cycle and SM), the softmax threads
// about half as long again for loads, dS, packing and stores, the four products 2048 cycles; an item takes 2750
// (exponentials, then the last half of dV and the next S behind each other).  Measured, with the MMA warp as it is now and
// before it stayed converged, and for attn_dkdv_split_kernel (P and dS through shared memory): 214, 233 and 275 us (one
// sequence of 4096, 32/8 heads of 128).
template <int HD>
struct DkvTmemSmem {
  static constexpr int QST = 2, DST = 2;
  static constexpr int THREADS = 64 + 256;
  static constexpr uint32_t TILE = BLK * HD * 2;
  static constexpr uint32_t K = 0, V = TILE, Q = 2 * TILE, DO = Q + QST * TILE;
  static constexpr uint32_t STATS = DO + DST * TILE;  // float [2 buffers][lse 128 | delta 128]
  static constexpr uint32_t BARS = STATS + 2 * 2 * BLK * 4;
  static constexpr uint32_t TOTAL = BARS + 256 + 1024;
};
enum DkvTmemBar {
  TK_KV_FULL = 0, TK_Q_FULL0 = 1, TK_Q_EMPTY0 = 3, TK_DO_FULL0 = 5, TK_DO_EMPTY0 = 7, TK_S_FULL = 9, TK_DP_FULL,
  TK_P_LO, TK_P_HI, TK_DS_LO, TK_DS_HI,  // P and dS of the first and of the last 64 query columns are stored
  TK_ACC_DONE, NUM_TK_BARS
};

// Column of k-step kk (16 of an item's 128 query columns) inside a 128-column region.  The thread of half h of a key row
// owns columns [32 h, 32 h + 32) and [64 + 32 h, 64 + 32 h + 32) and packs each 32 values into the first 16 of their columns.
__device__ __forceinline__ uint32_t dkv_kstep(uint32_t region, int kk) { return region + (kk >> 1) * 32 + (kk & 1) * 8; }

// Barrier over the 256 softmax threads of a group that tells all of them whether any passed `mine`.
__device__ __forceinline__ bool softmax_threads_any(int group, bool mine) {
  uint32_t any;
  asm volatile(
      "{\n\t"
      ".reg .pred p, q;\n\t"
      "setp.ne.u32 p, %1, 0;\n\t"
      "barrier.cta.red.or.pred.aligned q, %2, 256, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t"
      "}\n"
      : "=r"(any)
      : "r"(mine ? 1u : 0u), "r"(1 + group)
      : "memory");
  return any != 0;
}

template <int HD>
__global__ void __launch_bounds__(DkvTmemSmem<HD>::THREADS, 1)
attn_dkdv_tmem_kernel(const __grid_constant__ CUtensorMap tq, const __grid_constant__ CUtensorMap tk,
                      const __grid_constant__ CUtensorMap tv, const __grid_constant__ CUtensorMap tdo,
                      const float* __restrict__ LSE, const float* __restrict__ delta, __nv_bfloat16* __restrict__ dK,
                      __nv_bfloat16* __restrict__ dV, int S, int Hq, int Hkv, long long lddk, long long lddv, float scale,
                      float scale_log2, int* status) {
  using L = DkvTmemSmem<HD>;
  constexpr int QST = L::QST, DST = L::DST;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t* smem = smem_raw + (base - raw);
  const uint32_t bar0 = base + L::BARS;
  auto bar = [&](int i) { return bar0 + 8u * i; };
  volatile uint32_t* tmem_holder = reinterpret_cast<volatile uint32_t*>(smem + L::BARS + 8 * NUM_TK_BARS);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + L::BARS + 8 * NUM_TK_BARS + 8);
  float* stats = reinterpret_cast<float*>(smem + L::STATS);

  const int warp = uniform_warp_index(), lane = threadIdx.x & 31;
  const int n_tiles = (S + BLK - 1) / BLK;
  const int jt = blockIdx.x / Hkv;  // key tile; early key tiles have the most work and come first
  const int kv_head = blockIdx.x % Hkv, batch = blockIdx.y;
  const int G = Hq / Hkv;
  const int n_items = G * (n_tiles - jt);  // (query head of the group, query tile at or after the key tile)

  if (threadIdx.x == 0) {
    for (int i = 0; i < NUM_TK_BARS; ++i) mbar_init(bar(i), (i >= TK_P_LO && i < TK_ACC_DONE) ? 8 : 1);  // one arrival per softmax warp
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tq);
    tma_prefetch_desc(&tk);
    tma_prefetch_desc(&tv);
    tma_prefetch_desc(&tdo);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_holder)), 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_holder;
  // key rows on the lanes everywhere: S^T (later P^T) of item t, dP^T (later dS^T), the two accumulators
  const uint32_t t_st = tmem_base, t_dpt = tmem_base + 128u, t_dv = tmem_base + 256u, t_dk = t_dv + HD;

  if (warp == 0) {
    if (lane == 0) {
      mbar_expect_tx(bar(TK_KV_FULL), 2 * L::TILE);
      load_tile<HD>(base + L::K, &tk, bar(TK_KV_FULL), kv_head, jt * BLK, batch);
      load_tile<HD>(base + L::V, &tv, bar(TK_KV_FULL), kv_head, jt * BLK, batch);
      int it = jt, head = kv_head * G;
      for (int t = 0; t < n_items; ++t) {
        const int qs = t % QST, ds = t % DST;
        if (!mbar_wait(bar(TK_Q_EMPTY0 + qs), ((t / QST) & 1) ^ 1, abort_flag)) break;
        mbar_expect_tx(bar(TK_Q_FULL0 + qs), L::TILE);
        load_tile<HD>(base + L::Q + qs * L::TILE, &tq, bar(TK_Q_FULL0 + qs), head, it * BLK, batch);
        if (!mbar_wait(bar(TK_DO_EMPTY0 + ds), ((t / DST) & 1) ^ 1, abort_flag)) break;
        mbar_expect_tx(bar(TK_DO_FULL0 + ds), L::TILE);
        load_tile<HD>(base + L::DO + ds * L::TILE, &tdo, bar(TK_DO_FULL0 + ds), head, it * BLK, batch);
        if (++it == n_tiles) {
          it = jt;
          ++head;
        }
      }
    }
  } else if (warp == 1) {
    {
      const uint32_t leader = elect_one();
      constexpr uint32_t idesc_s = make_idesc_bf16(BLK, BLK, false, false);  // 128 keys x 128 queries
      constexpr uint32_t idesc_g = make_idesc_bf16(BLK, HD, false, true);
      // S^T = K Q^T of item t: the key tile is the A operand, so keys land on the lanes
      auto issue_s = [&](int t) -> bool {
        const int qs = t % QST;
        if (!mbar_wait_warp(bar(TK_Q_FULL0 + qs), (t / QST) & 1, abort_flag)) return false;
        tc_fence_after();
        const uint32_t sq = base + L::Q + qs * L::TILE;
#pragma unroll
        for (int k = 0; k < HD / 16; ++k) umma_bf16_elect(leader, t_st, kmajor_desc(base + L::K, k), kmajor_desc(sq, k), idesc_s, k != 0);
        umma_commit_elect(leader, bar(TK_S_FULL));
        return true;
      };
      auto issue_dp = [&](int t) -> bool {  // dP^T = V dO^T of item t
        const int ds = t % DST;
        if (!mbar_wait_warp(bar(TK_DO_FULL0 + ds), (t / DST) & 1, abort_flag)) return false;
        tc_fence_after();
        const uint32_t sdo = base + L::DO + ds * L::TILE;
#pragma unroll
        for (int k = 0; k < HD / 16; ++k) umma_bf16_elect(leader, t_dpt, kmajor_desc(base + L::V, k), kmajor_desc(sdo, k), idesc_s, k != 0);
        umma_commit_elect(leader, bar(TK_DP_FULL));
        return true;
      };
      // acc (+)= A B over the item's query rows [64 half, 64 half + 64): A = P^T or dS^T from tensor memory
      auto issue_grad = [&](uint32_t acc, uint32_t a_region, uint32_t b_tile, int t, int half) {
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
          const int k = half * 4 + kk;
          umma_bf16_ts_elect(leader, acc, dkv_kstep(a_region, k), mnmajor_desc(b_tile, k), idesc_g, (t | k) != 0);
        }
      };
      bool ok = mbar_wait_warp(bar(TK_KV_FULL), 0, abort_flag);
      if (ok && n_items > 0) ok = issue_s(0) && issue_dp(0);
      for (int t = 0; t < n_items && ok; ++t) {
        const int qs = t % QST, ds = t % DST;
        const uint32_t sq = base + L::Q + qs * L::TILE, sdo = base + L::DO + ds * L::TILE;
        if (!mbar_wait_warp(bar(TK_P_LO), t & 1, abort_flag)) { ok = false; break; }
        tc_fence_after();
        issue_grad(t_dv, t_st, sdo, t, 0);
        if (!mbar_wait_warp(bar(TK_P_HI), t & 1, abort_flag)) { ok = false; break; }
        tc_fence_after();
        issue_grad(t_dv, t_st, sdo, t, 1);
        umma_commit_elect(leader, bar(TK_DO_EMPTY0 + ds));
        // in order behind dV(t), which was the last reader of the region
        if (t + 1 < n_items && !issue_s(t + 1)) { ok = false; break; }
        if (!mbar_wait_warp(bar(TK_DS_LO), t & 1, abort_flag)) { ok = false; break; }
        tc_fence_after();
        issue_grad(t_dk, t_dpt, sq, t, 0);
        if (!mbar_wait_warp(bar(TK_DS_HI), t & 1, abort_flag)) { ok = false; break; }
        tc_fence_after();
        issue_grad(t_dk, t_dpt, sq, t, 1);
        umma_commit_elect(leader, bar(TK_Q_EMPTY0 + qs));
        if (t + 1 < n_items && !issue_dp(t + 1)) { ok = false; break; }
      }
      if (ok) umma_commit_elect(leader, bar(TK_ACC_DONE));
    }
  } else {
    const int q = warp & 3;
    const int hf = (warp - 2) >> 2;  // two threads per key row, each with 32 of the first and 32 of the last 64 query columns
    const int r = q * 32 + lane;     // key row inside the tile
    const int e = (warp - 2) * 32 + lane;  // 0..255: which statistic this thread fetches per item
    const uint32_t lane_addr = static_cast<uint32_t>(q * 32) << 16;
    bool ok = true;
    // statistic of a query tile for this thread's slot: log-sum-exp (slots 0..127) or delta (128..255) of one
    // query row; +inf as log-sum-exp of a row beyond the sequence turns its probabilities into zeros
    auto fetch_stat = [&](int head, int it) -> float {
      const int qrow = it * BLK + (e & 127);
      const long long at = (static_cast<long long>(batch) * Hq + head) * S + qrow;
      if (e < 128) return qrow < S ? LSE[at] : INFINITY;
      return qrow < S ? delta[at] : 0.f;
    };
    int it = jt, head = kv_head * G;
    float next_stat = fetch_stat(head, it);
    for (int t = 0; t < n_items; ++t) {
      const bool diag = it == jt;
      const int q_end = S - it * BLK;                  // query columns at or beyond this one do not exist
      const bool masked = diag || q_end < BLK;         // the same for the whole block
      float* my_stats = stats + (t & 1) * 2 * BLK;
      my_stats[e] = next_stat;
      if (++it == n_tiles) {
        it = jt;
        ++head;
      }
      if (t + 1 < n_items) next_stat = fetch_stat(head, it);  // travels while this item is processed
      ok = __all_sync(0xffffffffu, mbar_wait(bar(TK_S_FULL), t & 1, abort_flag)) && ok;
      // every statistic of this item is in shared memory; all threads leave together if one of them gave up
      ok = !softmax_threads_any(0, !ok);
      if (!ok) break;
      tc_fence_after();
      float p[2][32];
      {
        uint32_t sv[2][32];
#pragma unroll
        for (int h = 0; h < 2; ++h) tmem_ld_32x32(t_st + lane_addr + h * 64 + hf * 32, sv[h]);
        tmem_ld_wait();
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int c0 = h * 64 + hf * 32;
#pragma unroll
          for (int i4 = 0; i4 < 8; ++i4) {
            const float4 ls = *reinterpret_cast<const float4*>(my_stats + c0 + i4 * 4);
            const float lsv[4] = {ls.x, ls.y, ls.z, ls.w};
#pragma unroll
            for (int u = 0; u < 4; ++u) p[h][i4 * 4 + u] = fast_exp2(__uint_as_float(sv[h][i4 * 4 + u]) * scale_log2 - lsv[u]);
          }
          if (masked) {
#pragma unroll
            for (int i = 0; i < 32; ++i)  // causal: query column >= key row
              if ((diag && c0 + i < r) || c0 + i >= q_end) p[h][i] = 0.f;
          }
          uint32_t packed[16];
          pack32(p[h], packed);
          tmem_st_32x16(t_st + lane_addr + c0, packed);  // over score columns this thread has already read
          tmem_st_wait();
          tc_fence_before();
          __syncwarp();  // the lanes' stores are ordered before the one arrival of the warp
          if (lane == 0) mbar_arrive(bar(h == 0 ? TK_P_LO : TK_P_HI));
        }
      }
      ok = __all_sync(0xffffffffu, mbar_wait(bar(TK_DP_FULL), t & 1, abort_flag));  // acted upon at the next item's barrier
      tc_fence_after();
      {
        uint32_t dv[2][32];
#pragma unroll
        for (int h = 0; h < 2; ++h) tmem_ld_32x32(t_dpt + lane_addr + h * 64 + hf * 32, dv[h]);
        tmem_ld_wait();
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int c0 = h * 64 + hf * 32;
#pragma unroll
          for (int i4 = 0; i4 < 8; ++i4) {
            const float4 dl = *reinterpret_cast<const float4*>(my_stats + BLK + c0 + i4 * 4);
            const float dlv[4] = {dl.x, dl.y, dl.z, dl.w};
#pragma unroll
            for (int u = 0; u < 4; ++u) p[h][i4 * 4 + u] *= __uint_as_float(dv[h][i4 * 4 + u]) - dlv[u];
          }
          uint32_t packed[16];
          pack32(p[h], packed);
          tmem_st_32x16(t_dpt + lane_addr + c0, packed);
          tmem_st_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(bar(h == 0 ? TK_DS_LO : TK_DS_HI));
        }
      }
    }
    if (ok) {
      const bool done = mbar_wait(bar(TK_ACC_DONE), 0, abort_flag);
      if (__all_sync(0xffffffffu, done)) {
        tc_fence_after();
        const int krow = jt * BLK + r;
        const long long tok = static_cast<long long>(batch) * S + krow;
        store_acc<HD / 2>(t_dv + lane_addr + hf * (HD / 2), dV + tok * lddv + kv_head * HD + hf * (HD / 2), lddv, 1.f, S - krow);
        store_acc<HD / 2>(t_dk + lane_addr + hf * (HD / 2), dK + tok * lddk + kv_head * HD + hf * (HD / 2), lddk, scale, S - krow);
      }
    }
    tc_fence_before();
  }

  __syncthreads();
  if (*abort_flag) {
    const long long t0 = clock64();
    while (clock64() - t0 < 2000000LL) { }
    if (threadIdx.x == 0 && status) atomicCAS(status, 0, static_cast<int>(kTimeoutBarrier));
  }
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// ------------------------------------------------------------------ dK, dV at head dimension 64: two half pipelines
// Products are cheap here (1152 cycles an item) and the softmax threads set the pace, so two groups of eight warps take the
// two halves of every item's query columns, each with its own hand-over of P, dP and dS.  dP^T is computed per half
// (N = 64), so a half's region is free as soon as its own dK product has been issued, and the groups drift half an item
// apart: one forms dS (FMA, packing) under the exponentials (MUFU) of the other.  Tensor-core order per item t:
//
//   dV(t) half 0 | dK(t-1) half 1 | dP(t) half 1 | dV(t) half 1 | S(t+2) | dK(t) half 0 | dP(t+1) half 0
//
// Two sequences of 2048, 32/8 heads of 64, beside attn_dkdv_split_kernel on the same GPU: 88 us for 134; with the groups
// taking turns on whole items (one dP region makes dS, dK and the next dP a chain) 90 for 128; with sixteen warps on one item
// 101 for 138; with eight warps, before the MMA warp stayed converged, 104 for 129.
struct DkvHalves {
  static constexpr int HD = 64, QST = 4, DST = 3;
  static constexpr int THREADS = 64 + 512;
  static constexpr uint32_t TILE = BLK * HD * 2;
  static constexpr uint32_t K = 0, V = TILE, Q = 2 * TILE, DO = Q + QST * TILE;
  static constexpr uint32_t STATS = DO + DST * TILE;  // float [groups][2 buffers][lse 64 | delta 64]
  static constexpr uint32_t BARS = STATS + 2 * 2 * BLK * 4;
  static constexpr uint32_t TOTAL = BARS + 256 + 1024;
};
enum DkvHalvesBar {
  TH_KV_FULL = 0, TH_Q_FULL0 = 1, TH_Q_EMPTY0 = 5, TH_DO_FULL0 = 9, TH_DO_EMPTY0 = 12, TH_S_FULL0 = 15, TH_DP_FULL0 = 17,
  TH_P0 = 19, TH_DS0 = 21, TH_ACC_DONE = 23, NUM_TH_BARS = 24
};

__global__ void __launch_bounds__(DkvHalves::THREADS, 1)
attn_dkdv_halves_kernel(const __grid_constant__ CUtensorMap tq, const __grid_constant__ CUtensorMap tk,
                      const __grid_constant__ CUtensorMap tv, const __grid_constant__ CUtensorMap tdo,
                      const float* __restrict__ LSE, const float* __restrict__ delta, __nv_bfloat16* __restrict__ dK,
                      __nv_bfloat16* __restrict__ dV, int S, int Hq, int Hkv, long long lddk, long long lddv, float scale,
                      float scale_log2, int* status) {
  using L = DkvHalves;
  constexpr int HD = L::HD, QST = L::QST, DST = L::DST;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t* smem = smem_raw + (base - raw);
  const uint32_t bar0 = base + L::BARS;
  auto bar = [&](int i) { return bar0 + 8u * i; };
  volatile uint32_t* tmem_holder = reinterpret_cast<volatile uint32_t*>(smem + L::BARS + 8 * NUM_TH_BARS);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + L::BARS + 8 * NUM_TH_BARS + 8);
  float* stats = reinterpret_cast<float*>(smem + L::STATS);

  const int warp = uniform_warp_index(), lane = threadIdx.x & 31;
  const int n_tiles = (S + BLK - 1) / BLK;
  const int jt = blockIdx.x / Hkv;  // key tile; early key tiles have the most work and come first
  const int kv_head = blockIdx.x % Hkv, batch = blockIdx.y;
  const int G = Hq / Hkv;
  const int n_items = G * (n_tiles - jt);  // (query head of the group, query tile at or after the key tile)

  if (threadIdx.x == 0) {
    for (int i = 0; i < NUM_TH_BARS; ++i) mbar_init(bar(i), (i >= TH_P0 && i < TH_ACC_DONE) ? 8 : 1);  // one arrival per warp of a group
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tq);
    tma_prefetch_desc(&tk);
    tma_prefetch_desc(&tv);
    tma_prefetch_desc(&tdo);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_holder)), 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_holder;
  // key rows on the lanes everywhere: S^T (later P^T) of item t, dP^T (later dS^T), the two accumulators
  auto t_st = [&](int t) { return tmem_base + static_cast<uint32_t>(t & 1) * 128u; };
  const uint32_t t_dpt = tmem_base + 256u, t_dv = t_dpt + 128u, t_dk = t_dv + HD;

  if (warp == 0) {
    if (lane == 0) {
      mbar_expect_tx(bar(TH_KV_FULL), 2 * L::TILE);
      load_tile<HD>(base + L::K, &tk, bar(TH_KV_FULL), kv_head, jt * BLK, batch);
      load_tile<HD>(base + L::V, &tv, bar(TH_KV_FULL), kv_head, jt * BLK, batch);
      int it = jt, head = kv_head * G;
      for (int t = 0; t < n_items; ++t) {
        const int qs = t % QST, ds = t % DST;
        if (!mbar_wait(bar(TH_Q_EMPTY0 + qs), ((t / QST) & 1) ^ 1, abort_flag)) break;
        mbar_expect_tx(bar(TH_Q_FULL0 + qs), L::TILE);
        load_tile<HD>(base + L::Q + qs * L::TILE, &tq, bar(TH_Q_FULL0 + qs), head, it * BLK, batch);
        if (!mbar_wait(bar(TH_DO_EMPTY0 + ds), ((t / DST) & 1) ^ 1, abort_flag)) break;
        mbar_expect_tx(bar(TH_DO_FULL0 + ds), L::TILE);
        load_tile<HD>(base + L::DO + ds * L::TILE, &tdo, bar(TH_DO_FULL0 + ds), head, it * BLK, batch);
        if (++it == n_tiles) {
          it = jt;
          ++head;
        }
      }
    }
  } else if (warp == 1) {
    const uint32_t leader = elect_one();
    constexpr uint32_t idesc_s = make_idesc_bf16(BLK, BLK, false, false);  // 128 keys x 128 queries
    constexpr uint32_t idesc_dp = make_idesc_bf16(BLK, 64, false, false);  // 128 keys x 64 queries
    constexpr uint32_t idesc_g = make_idesc_bf16(BLK, HD, false, true);
    auto issue_s = [&](int t) -> bool {  // S^T = K Q^T of item t
      const int qs = t % QST;
      if (!mbar_wait_warp(bar(TH_Q_FULL0 + qs), (t / QST) & 1, abort_flag)) return false;
      tc_fence_after();
      const uint32_t sq = base + L::Q + qs * L::TILE;
#pragma unroll
      for (int k = 0; k < HD / 16; ++k) umma_bf16_elect(leader, t_st(t), kmajor_desc(base + L::K, k), kmajor_desc(sq, k), idesc_s, k != 0);
      umma_commit_elect(leader, bar(TH_S_FULL0 + (t & 1)));
      return true;
    };
    auto issue_dp = [&](int t, int half) -> bool {  // dP^T = V dO^T for the item's query rows [64 half, 64 half + 64)
      const int ds = t % DST;
      if (!mbar_wait_warp(bar(TH_DO_FULL0 + ds), (t / DST) & 1, abort_flag)) return false;
      tc_fence_after();
      const uint32_t sdo = base + L::DO + ds * L::TILE + half * 8192;
#pragma unroll
      for (int k = 0; k < HD / 16; ++k)
        umma_bf16_elect(leader, t_dpt + half * 64, kmajor_desc(base + L::V, k), kmajor_desc(sdo, k), idesc_dp, k != 0);
      umma_commit_elect(leader, bar(TH_DP_FULL0 + half));
      return true;
    };
    // acc (+)= A B over one half's query rows, once its group has stored A (P^T or dS^T) in tensor memory
    auto issue_grad = [&](int ready, int t, int half, uint32_t acc, uint32_t a_region, uint32_t b_tile) -> bool {
      if (!mbar_wait_warp(bar(ready + half), t & 1, abort_flag)) return false;
      tc_fence_after();
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) {
        const int k = half * 4 + kk;
        umma_bf16_ts_elect(leader, acc, dkv_kstep(a_region, k), mnmajor_desc(b_tile, k), idesc_g, (t | k) != 0);
      }
      return true;
    };
    auto q_tile = [&](int t) { return base + L::Q + (t % QST) * L::TILE; };
    auto do_tile = [&](int t) { return base + L::DO + (t % DST) * L::TILE; };
    auto last_of_item = [&](int t) -> bool {  // dK of the second half: the last reader of the item's Q
      if (!issue_grad(TH_DS0, t, 1, t_dk, t_dpt, q_tile(t))) return false;
      umma_commit_elect(leader, bar(TH_Q_EMPTY0 + t % QST));
      return true;
    };
    bool ok = mbar_wait_warp(bar(TH_KV_FULL), 0, abort_flag) && issue_s(0) && issue_dp(0, 0);
    if (ok && n_items > 1) ok = issue_s(1);
    for (int t = 0; t < n_items && ok; ++t) {
      ok = issue_grad(TH_P0, t, 0, t_dv, t_st(t), do_tile(t)) && (t == 0 || last_of_item(t - 1)) && issue_dp(t, 1) &&
           issue_grad(TH_P0, t, 1, t_dv, t_st(t), do_tile(t));
      if (!ok) break;
      umma_commit_elect(leader, bar(TH_DO_EMPTY0 + t % DST));
      // in order behind dV(t), which was the last reader of the region
      if (t + 2 < n_items && !issue_s(t + 2)) { ok = false; break; }
      ok = issue_grad(TH_DS0, t, 0, t_dk, t_dpt, q_tile(t)) && (t + 1 == n_items || issue_dp(t + 1, 0));
    }
    if (ok && last_of_item(n_items - 1)) umma_commit_elect(leader, bar(TH_ACC_DONE));
  } else {
    const int q = warp & 3;
    const int g = (warp - 2) >> 3;         // group: query columns [64 g, 64 g + 64) of every item
    const int gw = (warp - 2) & 7;         // warp inside the group
    const int hf = gw >> 2;                // two threads per key row, 32 columns each
    const int r = q * 32 + lane;           // key row inside the tile
    const int e = gw * 32 + lane;          // the first 128 fetch the statistics of the group's 64 query rows
    const uint32_t lane_addr = static_cast<uint32_t>(q * 32) << 16;
    const int c0 = g * 64 + hf * 32;       // first column of this thread
    bool ok = true;
    // log-sum-exp (slots 0..63) or delta (64..127) of one query row; +inf as log-sum-exp of a row beyond the sequence turns
    // its probabilities into zeros
    auto fetch_stat = [&](int head, int it) -> float {
      const int qrow = it * BLK + g * 64 + (e & 63);
      const long long at = (static_cast<long long>(batch) * Hq + head) * S + qrow;
      if (e < 64) return qrow < S ? LSE[at] : INFINITY;
      return qrow < S ? delta[at] : 0.f;
    };
    int it = jt, head = kv_head * G;
    float next_stat = e < 128 ? fetch_stat(head, it) : 0.f;
    for (int t = 0; t < n_items; ++t) {
      const bool diag = it == jt;
      const int q_end = S - it * BLK;                  // query columns at or beyond this one do not exist
      const bool masked = diag || q_end < BLK;         // the same for the whole block
      float* my_stats = stats + (g * 2 + (t & 1)) * BLK;
      if (e < 128) my_stats[e] = next_stat;
      if (++it == n_tiles) {
        it = jt;
        ++head;
      }
      if (t + 1 < n_items && e < 128) next_stat = fetch_stat(head, it);  // travels while this item is processed
      ok = mbar_wait_warp(bar(TH_S_FULL0 + (t & 1)), (t >> 1) & 1, abort_flag) && ok;
      // every statistic of this item is in shared memory; all threads of the group leave together if one of them gave up
      ok = !softmax_threads_any(g, !ok);
      if (!ok) break;
      tc_fence_after();
      float p[32];
      {
        uint32_t sv[32];
        tmem_ld_32x32(t_st(t) + lane_addr + c0, sv);
        tmem_ld_wait();
#pragma unroll
        for (int i4 = 0; i4 < 8; ++i4) {
          const float4 ls = *reinterpret_cast<const float4*>(my_stats + hf * 32 + i4 * 4);
          const float lsv[4] = {ls.x, ls.y, ls.z, ls.w};
#pragma unroll
          for (int u = 0; u < 4; ++u) p[i4 * 4 + u] = fast_exp2(__uint_as_float(sv[i4 * 4 + u]) * scale_log2 - lsv[u]);
        }
        if (masked) {
#pragma unroll
          for (int i = 0; i < 32; ++i)  // causal: query column >= key row
            if ((diag && c0 + i < r) || c0 + i >= q_end) p[i] = 0.f;
        }
        uint32_t packed[16];
        pack32(p, packed);
        tmem_st_32x16(t_st(t) + lane_addr + c0, packed);  // over score columns this thread has already read
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();  // the lanes' stores are ordered before the one arrival of the warp
        if (lane == 0) mbar_arrive(bar(TH_P0 + g));
      }
      ok = mbar_wait_warp(bar(TH_DP_FULL0 + g), t & 1, abort_flag);  // acted upon at the next item's barrier
      tc_fence_after();
      {
        uint32_t dv[32];
        tmem_ld_32x32(t_dpt + lane_addr + c0, dv);
        tmem_ld_wait();
#pragma unroll
        for (int i4 = 0; i4 < 8; ++i4) {
          const float4 dl = *reinterpret_cast<const float4*>(my_stats + 64 + hf * 32 + i4 * 4);
          const float dlv[4] = {dl.x, dl.y, dl.z, dl.w};
#pragma unroll
          for (int u = 0; u < 4; ++u) p[i4 * 4 + u] *= __uint_as_float(dv[i4 * 4 + u]) - dlv[u];
        }
        uint32_t packed[16];
        pack32(p, packed);
        tmem_st_32x16(t_dpt + lane_addr + c0, packed);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(TH_DS0 + g));
      }
    }
    if (ok && mbar_wait_warp(bar(TH_ACC_DONE), 0, abort_flag)) {
      tc_fence_after();
      const int krow = jt * BLK + r, col = hf * (HD / 2);
      const long long tok = static_cast<long long>(batch) * S + krow;
      if (g == 0)
        store_acc<HD / 2>(t_dv + lane_addr + col, dV + tok * lddv + kv_head * HD + col, lddv, 1.f, S - krow);
      else
        store_acc<HD / 2>(t_dk + lane_addr + col, dK + tok * lddk + kv_head * HD + col, lddk, scale, S - krow);
    }
    tc_fence_before();
  }

  __syncthreads();
  if (*abort_flag) {
    const long long t0 = clock64();
    while (clock64() - t0 < 2000000LL) { }
    if (threadIdx.x == 0 && status) atomicCAS(status, 0, static_cast<int>(kTimeoutBarrier));
  }
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

template <int HD>
int launch_dkdv_tmem(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& tdo,
                     const float* lse, const float* delta, void* dk, void* dv, int B, int S, int Hq, int Hkv,
                     long long lddk, long long lddv, float scale, int* status, cudaStream_t stream) {
  const int n_tiles = (S + BLK - 1) / BLK;
  const dim3 grid(n_tiles * Hkv, B, 1);
  static bool configured = false;
  if constexpr (HD == 64) {
    if (!configured) {
      const cudaError_t e = cudaFuncSetAttribute(attn_dkdv_halves_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, DkvHalves::TOTAL);
      if (e != cudaSuccess) return static_cast<int>(e);
      configured = true;
    }
    attn_dkdv_halves_kernel<<<grid, DkvHalves::THREADS, DkvHalves::TOTAL, stream>>>(
        tq, tk, tv, tdo, lse, delta, static_cast<__nv_bfloat16*>(dk), static_cast<__nv_bfloat16*>(dv), S, Hq, Hkv, lddk,
        lddv, scale, scale * 1.4426950408889634f, status);
  } else {
    if (!configured) {
      const cudaError_t e = cudaFuncSetAttribute(attn_dkdv_tmem_kernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 DkvTmemSmem<HD>::TOTAL);
      if (e != cudaSuccess) return static_cast<int>(e);
      configured = true;
    }
    attn_dkdv_tmem_kernel<HD><<<grid, DkvTmemSmem<HD>::THREADS, DkvTmemSmem<HD>::TOTAL, stream>>>(
        tq, tk, tv, tdo, lse, delta, static_cast<__nv_bfloat16*>(dk), static_cast<__nv_bfloat16*>(dv), S, Hq, Hkv, lddk,
        lddv, scale, scale * 1.4426950408889634f, status);
  }
  return static_cast<int>(cudaGetLastError());
}

template <int HD>
int launch_bwd_tmem(const void* dout, const void* q, const void* k, const void* v, const void* o, const float* lse,
                    float* delta, void* dq, void* dk, void* dv, int B, int S, int Hq, int Hkv, long long ldq,
                    long long ldk, long long ldv, long long lddq, long long lddk, long long lddv, float scale, int* status,
                    cudaStream_t stream, int parts) {
  CUtensorMap tq, tk, tv, tdo;
  if (!make_attn_tensormap(&tq, q, HD, Hq, S, B, ldq)) return -2;
  if (!make_attn_tensormap(&tk, k, HD, Hkv, S, B, ldk)) return -3;
  if (!make_attn_tensormap(&tv, v, HD, Hkv, S, B, ldv)) return -4;
  if (!make_attn_tensormap(&tdo, dout, HD, Hq, S, B, static_cast<long long>(Hq) * HD)) return -5;
  cudaGetLastError();
  if (parts & 1) launch_delta<HD>(o, dout, delta, B, S, Hq, stream);
  int rc = 0;
  if (parts & 2) rc = launch_dkdv_tmem<HD>(tq, tk, tv, tdo, lse, delta, dk, dv, B, S, Hq, Hkv, lddk, lddv, scale, status, stream);
  if (rc == 0 && (parts & 4)) rc = launch_dq_tmem<HD>(tq, tk, tv, tdo, lse, delta, dq, B, S, Hq, Hkv, lddq, scale, status, stream);
  return rc;
}

}  // namespace attn
}  // namespace tft

// dQ alone (delta must have been computed): the dQ kernel of this file, for use behind the dK/dV kernel
// of attention_bwd.cu or of this file.  Arguments as the corresponding ones of tft_attn_bwd.
TFT_API int tft_attn_dq_tmem(const void* dout, const void* q, const void* k, const void* v, const float* lse,
                             const float* delta, void* dq, int B, int S, int Hq, int Hkv, int hd, int ldq, int ldk,
                             int ldv, int lddq, float scale, int* status, cudaStream_t stream) {
  using namespace tft::attn;
  if (Hq % Hkv || (ldq % 8) || (ldk % 8) || (ldv % 8) || (lddq % 8)) return -1;
  CUtensorMap tq, tk, tv, tdo;
  if (!make_attn_tensormap(&tq, q, hd, Hq, S, B, ldq)) return -2;
  if (!make_attn_tensormap(&tk, k, hd, Hkv, S, B, ldk)) return -3;
  if (!make_attn_tensormap(&tv, v, hd, Hkv, S, B, ldv)) return -4;
  if (!make_attn_tensormap(&tdo, dout, hd, Hq, S, B, static_cast<long long>(Hq) * hd)) return -5;
  cudaGetLastError();
  if (hd == 128) return launch_dq_tmem<128>(tq, tk, tv, tdo, lse, delta, dq, B, S, Hq, Hkv, lddq, scale, status, stream);
  if (hd == 64) return launch_dq_tmem<64>(tq, tk, tv, tdo, lse, delta, dq, B, S, Hq, Hkv, lddq, scale, status, stream);
  return -1;
}

// Causal attention backward with P and dS in tensor memory: same contract as tft_attn_bwd
// (attention_bwd.cu); parts = 1 (delta) | 2 (dK/dV) | 4 (dQ) selects kernels, 7 runs all three.
TFT_API int tft_attn_bwd_tmem(const void* dout, const void* q, const void* k, const void* v, const void* o,
                              const float* lse, float* delta, void* dq, void* dk, void* dv, int B, int S, int Hq,
                              int Hkv, int hd, int ldq, int ldk, int ldv, int lddq, int lddk, int lddv, float scale,
                              int* status, cudaStream_t stream, int parts) {
  using namespace tft::attn;
  if (Hq % Hkv || (ldq % 8) || (ldk % 8) || (ldv % 8) || (lddq % 8) || (lddk % 8) || (lddv % 8)) return -1;
  if (hd == 128)
    return launch_bwd_tmem<128>(dout, q, k, v, o, lse, delta, dq, dk, dv, B, S, Hq, Hkv, ldq, ldk, ldv, lddq, lddk, lddv,
                                scale, status, stream, parts);
  if (hd == 64)
    return launch_bwd_tmem<64>(dout, q, k, v, o, lse, delta, dq, dk, dv, B, S, Hq, Hkv, ldq, ldk, ldv, lddq, lddk, lddv,
                               scale, status, stream, parts);
  return -1;
}
