// A whole sequence of dependent batched products in ONE launch (sm_100a).
//
// Newton-Schulz on a small or medium matrix is eighteen products of a few
// microseconds each.  As separate launches every product pays the launch, the
// ramp of a persistent kernel (barriers, TMEM, descriptor fetch) and an empty
// last wave, and the host cannot issue them fast enough.  Here the products are
// a list of tiles in dependency order.  CTAs draw tiles from a ticket counter;
// a tile of matrix b starts when `done[b]` (warps that finished a tile of that
// matrix) has reached the count of everything its product needs.  Matrices of a
// batch, and batches of different shapes, run past each other without a barrier.
//
// Progress needs no co-residency of the CTAs: tickets are handed out in list
// order, a tile only depends on tiles with smaller tickets, and those have been
// drawn by CTAs that are already running and whose own waits point further back.
// So the launch is an ordinary one and may share the GPU with kernels of other
// streams that hold some of the SMs.
//
// Per CTA the roles are those of the stand-alone GEMM (TMA producer, MMA issuer,
// epilogue warps with two TMEM accumulators); the producer also draws the
// tickets and hands the entries to the other roles through a four-slot ring.
// A product with few tiles and a long inner dimension (Gram of a flat matrix) is
// split over K: each split stores an fp32 partial tile, and a sum entry adds them
// in a fixed order, so results do not depend on timing.
//
// What bounds it: small batches, the chain load -> MMA -> store -> flag -> load;
// many tiles, the L2 -> SM stream of a 128 x BN tile (16 KB + BN * 128 bytes per
// k-block at 64 B/clk/SM).
#include <cuda.h>
#include <cuda_runtime.h>
#include <string.h>

#include "chain_sm100.cuh"
#include "gemm_epilogue.cuh"
#include "ptx_sm100.cuh"
#include "tensor_map.cuh"

namespace dmuon {
void count_launch();

namespace {

template <int BN>
struct ChainCfg {
  static constexpr int kStages = (BN == 64) ? 8 : 6;
  static constexpr int kABytes = BM * BK * 2;
  static constexpr int kBBytes = BN * BK * 2;
  static constexpr int kStageBytes = kABytes + kBBytes;
  static constexpr int kTmemCols = 2 * BN;
};

constexpr int kRing = 4;
// Eight epilogue warps, two per TMEM lane quarter with half of the columns each: in a chain of
// small products the time from a tile's last MMA to its flag is paid once per product.
constexpr int kEpiWarps = 8;
constexpr int kChainThreads = 64 + 32 * kEpiWarps;
constexpr int kSumCols = 64;        // a sum entry covers 128 x 64 elements

// An operation as the kernel keeps it in shared memory.
struct OpS {
  KParams k;
  const float* partials;
  int map_a, map_b, kb_per_split, splits;
};

// Launch parameters.  The tensor maps travel in them: maps in global memory that the host
// fills by copy need a proxy fence on each map by the thread that issues the loads, in every
// CTA, or a descriptor cached for an earlier owner of the address may be used.
struct ChainParams {
  CUtensorMap maps[DMUON_CHAIN_MAX_MAPS];
  DmuonChainFinal fin[DMUON_CHAIN_MAX_GROUPS];
  const DmuonChainOp* ops;
  const int4* tab;
  int* counters;
  char* work;
  int* status;
  int n_ops, n_maps, total, n_counters;
};
static_assert(sizeof(ChainParams) <= 32764, "kernel parameters are limited to 32,764 bytes");

constexpr int kBarBytes = 512;
constexpr int kStageBytesAll = kEpiWarps * kStageWarpBytes;
template <int BN>
constexpr int chain_smem_bytes(int n_ops) {
  return ChainCfg<BN>::kStages * ChainCfg<BN>::kStageBytes + kBarBytes + kStageBytesAll + n_ops * static_cast<int>(sizeof(OpS)) + 1024;
}

// A list entry: x = op | mirror << 8 | split << 16, y = row tile | column tile << 16,
// z = matrix within the batch | counter << 16, w = value the counter has to reach first.
__device__ __forceinline__ int entry_op(const int4& e) { return e.x & 0xff; }
__device__ __forceinline__ bool entry_mirror(const int4& e) { return (e.x >> 8) & 1; }
__device__ __forceinline__ int entry_split(const int4& e) { return (e.x >> 16) & 0x7fff; }
__device__ __forceinline__ int entry_m(const int4& e) { return e.y & 0xffff; }
__device__ __forceinline__ int entry_n(const int4& e) { return (e.y >> 16) & 0xffff; }
__device__ __forceinline__ int entry_b(const int4& e) { return e.z & 0xffff; }
__device__ __forceinline__ int entry_ctr(const int4& e) { return (e.z >> 16) & 0xffff; }

__device__ __forceinline__ void entry_k_range(const OpS& op, const int4& e, int& kb0, int& kb1) {
  const int num_kb = (op.k.K + BK - 1) / BK;
  kb0 = 0;
  kb1 = num_kb;
  if (op.kb_per_split > 0) {
    kb0 = entry_split(e) * op.kb_per_split;
    kb1 = min(num_kb, kb0 + op.kb_per_split);
  }
}

template <typename T>
__device__ __forceinline__ T* work_at(const ChainParams& p, long long offset) {
  return offset < 0 ? nullptr : reinterpret_cast<T*>(p.work + offset);
}

__device__ __forceinline__ void build_op(OpS& s, const DmuonChainOp& o, const ChainParams& p) {
  KParams k = {};
  k.M = o.M; k.N = o.N; k.K = o.K;
  k.a_mn_major = o.a_mn_major; k.b_mn_major = o.b_mn_major; k.ab_fp16 = o.ab_fp16;
  k.alpha = o.alpha; k.beta = o.beta; k.diag = o.diag;
  k.alpha_vec = work_at<const float>(p, o.alpha_vec);
  k.C = work_at<const void>(p, o.C); k.D = work_at<void>(p, o.D);
  k.ldc = o.ldc; k.ldd = o.ldd;
  k.strideC = o.strideC; k.strideD = o.strideD;
  k.out_kind = o.out_kind;
  if (o.final_slot >= 0) {
    const DmuonChainFinal& f = p.fin[o.final_slot];
    k.C = f.C; k.D = f.D;
    k.C_tab = f.C_tab; k.D_tab = f.D_tab; k.D2_tab = f.D2_tab;
    k.alpha_vec = f.alpha_vec;
    k.ldc = f.ldc; k.ldd = f.ldd; k.ldd2 = f.ldd2;
    k.strideC = f.strideC; k.strideD = f.strideD;
    k.alpha = f.alpha; k.beta = f.beta;
    k.out_kind = f.out_kind;
  }
  if (k.C == nullptr && k.C_tab == nullptr) k.beta = 0.f;
  s.k = k;
  s.partials = work_at<const float>(p, o.partials);
  s.map_a = o.map_a; s.map_b = o.map_b;
  s.kb_per_split = o.kb_per_split; s.splits = o.splits;
}

// Spin until `*count` reaches `want`: in a short chain the pause of a sleeping poll
// would be a good part of a product.
__device__ __forceinline__ bool wait_count(const int* count, int want, volatile int* abort_flag) {
  if (ld_acquire_gpu(count) >= want) return true;
  const long long t0 = clock64();
  uint32_t spins = 0;
  while (true) {
    if (ld_acquire_gpu(count) >= want) return true;
    if ((++spins & 63u) == 0u) {
      if (*abort_flag) return false;
      if (clock64() - t0 > kWaitBudgetCycles) {
        *abort_flag = 1;
        return false;
      }
    }
  }
}

template <int BN>
__global__ void __launch_bounds__(kChainThreads, 1) chain_kernel(const __grid_constant__ ChainParams p) {
  using C = ChainCfg<BN>;
  constexpr int S = C::kStages;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* sA = smem;
  uint8_t* sB = smem + S * C::kABytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + S * C::kStageBytes);
  const uint32_t full0 = smem_u32(bars);
  const uint32_t empty0 = smem_u32(bars + S);
  const uint32_t tfull0 = smem_u32(bars + 2 * S);
  const uint32_t tempty0 = smem_u32(bars + 2 * S + 2);
  const uint32_t rfull0 = smem_u32(bars + 2 * S + 4);
  const uint32_t rempty0 = smem_u32(bars + 2 * S + 4 + kRing);
  int4* ring = reinterpret_cast<int4*>(bars + 2 * S + 4 + 2 * kRing);     // 28 * 8 bytes in: 16-byte aligned
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(ring + kRing);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  uint8_t* staging = smem + S * C::kStageBytes + kBarBytes;
  OpS* ops = reinterpret_cast<OpS*>(staging + kStageBytesAll);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  int* const ticket = p.counters;
  int* const exits = p.counters + 1;
  int* const done = p.counters + 2;

  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(full0 + 8 * s, 1);
      mbar_init(empty0 + 8 * s, 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(tfull0 + 8 * a, 1);
      mbar_init(tempty0 + 8 * a, kEpiWarps);
    }
    for (int i = 0; i < kRing; ++i) {
      mbar_init(rfull0 + 8 * i, 1);
      mbar_init(rempty0 + 8 * i, 1 + kEpiWarps);     // MMA issuer and epilogue warps
    }
    *abort_flag = 0;
    fence_barrier_init();
    fence_proxy_async_smem();
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), C::kTmemCols);
    tmem_relinquish();
  }
  for (int i = threadIdx.x; i < p.n_ops; i += kChainThreads) build_op(ops[i], p.ops[i], p);
  for (int i = threadIdx.x; i < p.n_maps; i += kChainThreads) tma_prefetch_desc(p.maps + i);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  int fail_code = 0;

  if (warp == 0) {
    if (lane == 0) {
      // ---------------- tickets and TMA ----------------
      int stage = 0;
      uint32_t phase = 0;
      uint32_t cnt = 0;
      int t = atomicAdd(ticket, 1);
      bool ok = true;
      while (ok) {
        const uint32_t slot = cnt % kRing;
        if (!mbar_wait_bounded(rempty0 + 8 * slot, ((cnt / kRing) & 1u) ^ 1u, abort_flag)) {
          fail_code = kStatusTimeoutProducer;
          break;
        }
        int4 e = make_int4(-1, 0, 0, 0);
        if (t < p.total) e = __ldg(p.tab + t);
        ring[slot] = e;
        mbar_arrive(rfull0 + 8 * slot);
        ++cnt;
        if (e.x < 0) break;
        const OpS& op = ops[entry_op(e)];
        if (e.w > 0) {
          if (!wait_count(done + entry_ctr(e), e.w, abort_flag)) {
            fail_code = kStatusTimeoutChain;
            break;
          }
          fence_proxy_async_global();      // other CTAs' stores before this thread's bulk loads
        }
        // The next ticket is drawn now that this tile can run, and its latency hides behind the loads.
        // Drawn before the wait, a CTA would sit on two tiles of a product while others idle
        // (1024 x 1024: 252 us for the chain).
        t = atomicAdd(ticket, 1);
        if (op.map_a < 0) continue;        // a sum: the epilogue warps do all of it
        const CUtensorMap* tmA = p.maps + op.map_a;
        const CUtensorMap* tmB = p.maps + op.map_b;
        const int m0 = entry_m(e) * BM, n0 = entry_n(e) * BN, b = entry_b(e);
        const int a_mn = op.k.a_mn_major, b_mn = op.k.b_mn_major;
        int kb, kb1;
        entry_k_range(op, e, kb, kb1);
        for (; kb < kb1; ++kb) {
          if (!mbar_wait_bounded(empty0 + 8 * stage, phase ^ 1u, abort_flag)) {
            ok = false;
            fail_code = kStatusTimeoutProducer;
            break;
          }
          const uint32_t fb = full0 + 8 * stage;
          mbar_arrive_expect_tx(fb, C::kStageBytes);
          const uint32_t a_dst = smem_u32(sA + stage * C::kABytes);
          const uint32_t b_dst = smem_u32(sB + stage * C::kBBytes);
          if (!a_mn) {
            tma_load_3d(a_dst, tmA, fb, kb * BK, m0, b);
          } else {
#pragma unroll
            for (int mb = 0; mb < BM / 64; ++mb)
              tma_load_3d(a_dst + mb * kBlockBytes, tmA, fb, m0 + 64 * mb, kb * BK, b);
          }
          if (!b_mn) {
            tma_load_3d(b_dst, tmB, fb, kb * BK, n0, b);
          } else {
#pragma unroll
            for (int nb = 0; nb < BN / 64; ++nb)
              tma_load_3d(b_dst + nb * kBlockBytes, tmB, fb, n0 + 64 * nb, kb * BK, b);
          }
          if (++stage == S) {
            stage = 0;
            phase ^= 1u;
          }
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      // ---------------- MMA issuer ----------------
      int stage = 0;
      uint32_t phase = 0;
      int acc = 0;
      uint32_t acc_phase = 0;
      bool ok = true;
      for (uint32_t cnt = 0; ok; ++cnt) {
        const uint32_t slot = cnt % kRing;
        if (!mbar_wait_bounded(rfull0 + 8 * slot, (cnt / kRing) & 1u, abort_flag)) {
          fail_code = kStatusTimeoutMma;
          break;
        }
        const int4 e = ring[slot];
        mbar_arrive(rempty0 + 8 * slot);
        if (e.x < 0) break;
        const OpS& op = ops[entry_op(e)];
        if (op.map_a < 0) continue;
        if (!mbar_wait_bounded(tempty0 + 8 * acc, acc_phase ^ 1u, abort_flag)) {
          fail_code = kStatusTimeoutMma;
          break;
        }
        tc_fence_after_sync();
        const int a_mn = op.k.a_mn_major, b_mn = op.k.b_mn_major;
        const uint32_t idesc = make_idesc_f16(BM, BN, op.k.ab_fp16 != 0, a_mn != 0, b_mn != 0);
        const uint32_t d_tmem = tmem_base + static_cast<uint32_t>(acc * BN);
        int kb0, kb1;
        entry_k_range(op, e, kb0, kb1);
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait_bounded(full0 + 8 * stage, phase, abort_flag)) {
            ok = false;
            fail_code = kStatusTimeoutMma;
            break;
          }
          tc_fence_after_sync();
          const uint32_t a_base = smem_u32(sA + stage * C::kABytes);
          const uint32_t b_base = smem_u32(sB + stage * C::kBBytes);
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k) {
            const uint64_t adesc = a_mn ? make_smem_desc_sw128(a_base + k * 2048, kBlockBytes, 1024)
                                        : make_smem_desc_sw128(a_base + k * 32, 16, 1024);
            const uint64_t bdesc = b_mn ? make_smem_desc_sw128(b_base + k * 2048, kBlockBytes, 1024)
                                        : make_smem_desc_sw128(b_base + k * 32, 16, 1024);
            umma_f16_ss(d_tmem, adesc, bdesc, idesc, (kb != kb0 || k != 0) ? 1u : 0u);
          }
          umma_commit(empty0 + 8 * stage);
          if (++stage == S) {
            stage = 0;
            phase ^= 1u;
          }
        }
        if (!ok) break;
        umma_commit(tfull0 + 8 * acc);
        acc ^= 1;
        if (acc == 0) acc_phase ^= 1u;
      }
    }
  } else {
    // ---------------- epilogue (warps 2..9) ----------------
    const int q = warp & 3;              // TMEM lane quarter this warp may read
    const int half = (warp - 2) >> 2;    // which half of the tile's columns
    uint8_t* const stage_mem = staging + (warp - 2) * kStageWarpBytes;
    int acc = 0;
    uint32_t acc_phase = 0;
    for (uint32_t cnt = 0;; ++cnt) {
      const uint32_t slot = cnt % kRing;
      // a wait that gave up ends the whole warp: the TMEM loads below need all its lanes
      if (!__all_sync(0xffffffffu, mbar_wait_bounded(rfull0 + 8 * slot, (cnt / kRing) & 1u, abort_flag))) {
        fail_code = kStatusTimeoutEpilogue;
        break;
      }
      const int4 e = ring[slot];
      __syncwarp();
      if (lane == 0) mbar_arrive(rempty0 + 8 * slot);
      if (e.x < 0) break;
      const OpS& op = ops[entry_op(e)];
      const bool product = op.map_a >= 0;
      const int b = entry_b(e);
      const int row0 = entry_m(e) * BM + q * 32;
      const TileEpilogue tile(op.k, op.kb_per_split > 0 ? b * op.splits + entry_split(e) : b, row0,
                                    entry_mirror(e), stage_mem, lane);
      if (e.w > 0 && (tile.add_c || !product)) {
        // what other CTAs stored is read here: one lane acquires for the warp, the reads go to L2
        bool ready = true;
        if (lane == 0) ready = wait_count(done + entry_ctr(e), e.w, abort_flag);
        if (!ready) fail_code = kStatusTimeoutChain;
        if (!__all_sync(0xffffffffu, ready)) break;
      }
      if (product) {
        const int col0 = entry_n(e) * BN + half * (BN / 2);
        RawC c;
        tile.fetch_c(c, col0);           // arrives while the product runs
        if (!__all_sync(0xffffffffu, mbar_wait_bounded(tfull0 + 8 * acc, acc_phase, abort_flag))) {
          fail_code = kStatusTimeoutEpilogue;
          break;
        }
        tc_fence_after_sync();
        tile.run(tmem_base + (static_cast<uint32_t>(q * 32) << 16) + static_cast<uint32_t>(acc * BN + half * (BN / 2)),
                 col0, BN / 2, c);
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(tempty0 + 8 * acc);
        acc ^= 1;
        if (acc == 0) acc_phase ^= 1u;
      } else {
        // sum of the partial products, in the order of the splits
        const int col0 = entry_n(e) * kSumCols + half * 32;
        const int row = row0 + lane;
        if (col0 < op.k.N) {
          float v[32];
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = 0.f;
          if (row < op.k.M) {
            const long long plane = static_cast<long long>(op.k.M) * op.k.N;
            const float* src = op.partials + static_cast<long long>(b) * op.splits * plane +
                               static_cast<long long>(row) * op.k.N + col0;
            const int nvec = min(32, op.k.N - col0) / 4;     // N is a multiple of 8
            for (int s = 0; s < op.splits; ++s, src += plane) {
#pragma unroll
              for (int i = 0; i < 8; ++i) {
                if (i < nvec) {
                  const float4 x = __ldcg(reinterpret_cast<const float4*>(src) + i);
                  v[4 * i] += x.x;
                  v[4 * i + 1] += x.y;
                  v[4 * i + 2] += x.z;
                  v[4 * i + 3] += x.w;
                }
              }
            }
          }
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] *= tile.alpha;
          RawC c;
          tile.fetch_c(c, col0);
          tile.store(v, c, col0);
        }
      }
      // The release covers the stores of the whole warp; who loads them through the async
      // proxy fences after its acquire.
      __syncwarp();
      if (lane == 0) red_add_release_gpu(done + entry_ctr(e), 1);
    }
  }

  // ---------------- teardown ----------------
  tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag) {
    if (fail_code != 0 && p.status != nullptr) atomicCAS(p.status, 0, fail_code);
    // bulk copies that may still be in flight land before the shared memory is handed on
    for (int i = 0; i < 64; ++i) __nanosleep(2000);
    __syncthreads();
  }
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, C::kTmemCols);
  }
  if (warp == 0) {
    // the last CTA to leave clears the counters for the next launch: nobody waits on them any more
    int last = 0;
    if (lane == 0) {
      __threadfence();
      last = atomicAdd(exits, 1) == static_cast<int>(gridDim.x) - 1;
    }
    if (__shfl_sync(0xffffffffu, last, 0)) {
      for (int i = lane; i < p.n_counters; i += 32) p.counters[i] = 0;
    }
  }
}

// ---- CTA pairs (cta_group::2) --------------------------------------------------------
//
// Same list, same counters; an entry is a tile of 256 rows that two CTAs of a cluster
// share (128 rows each, MMAs issued by the leader).  The leader's producer draws the
// tickets and writes every entry into both CTAs' rings.  For lists whose products fill
// the GPU; no split over K, there are tiles enough.
//
// What bounds it is the L2 -> SM stream, which delivers about 80 bytes per nanosecond to
// an SM (302 ns per 24 KB k-block on an otherwise idle GPU with every stage free): with
// 256 columns a CTA pulls 32 KB per k-block for 512 clocks of MMA.
//
// WIDE: an entry is one or two such tiles side by side.  Two share their A rows, 48 KB
// for 1024 clocks.  Both fill the tensor memory, so the next entry cannot use a second
// accumulator set; instead the halves run out of step by the depth of the stage ring: the
// last k-blocks of an entry are done for half 0 first, then for half 1, and so are the
// first ones of the next entry.  While one half runs, the epilogue drains the other.
// Pays for long lists only (choose_wide in ops/chain.py has the line and the figures).
template <bool WIDE>
struct PairCfg {
  static constexpr int kStages = WIDE ? 4 : 6;
  static constexpr int kABytes = BM * BK * 2;            // 128 rows per CTA
  static constexpr int kBBytes = 128 * BK * 2;           // 128 of the 256 columns of a half per CTA
  static constexpr int kHalves = WIDE ? 2 : 1;
  static constexpr int kStageBytes = kABytes + kHalves * kBBytes;
};
constexpr int kPairBN = 256;
template <bool WIDE>
constexpr int pair_smem_bytes(int n_ops) {
  return PairCfg<WIDE>::kStages * PairCfg<WIDE>::kStageBytes + kBarBytes + kStageBytesAll +
         n_ops * static_cast<int>(sizeof(OpS)) + 1024;
}

// flags of a wide entry: bit 8 / 10 = mirror half 0 / 1, bit 9 = there is a half 1
template <bool WIDE>
__device__ __forceinline__ int entry_halves(const int4& e) { return WIDE ? 1 + ((e.x >> 9) & 1) : 1; }
__device__ __forceinline__ bool entry_mirror_half(const int4& e, int h) { return (e.x >> (8 + 2 * h)) & 1; }

template <bool WIDE>
__global__ void __launch_bounds__(kChainThreads, 1) chain_pair_kernel(const __grid_constant__ ChainParams p) {
  using C = PairCfg<WIDE>;
  constexpr int S = C::kStages;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* sA = smem;
  uint8_t* sB = smem + S * C::kABytes;              // per stage: half 0, then half 1
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + S * C::kStageBytes);
  const uint32_t full0 = smem_u32(bars);
  const uint32_t empty0 = smem_u32(bars + S);
  const uint32_t tfull0 = smem_u32(bars + 2 * S);
  const uint32_t tempty0 = smem_u32(bars + 2 * S + 2);
  const uint32_t rfull0 = smem_u32(bars + 2 * S + 4);
  const uint32_t rempty0 = smem_u32(bars + 2 * S + 4 + kRing);
  int4* ring = reinterpret_cast<int4*>(bars + 2 * S + 4 + 2 * kRing);     // an even number of 8-byte words in
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(ring + kRing);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  uint8_t* staging = smem + S * C::kStageBytes + kBarBytes;
  OpS* ops = reinterpret_cast<OpS*>(staging + kStageBytesAll);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();          // 0 = leader
  const bool leader = rank == 0;
  int* const ticket = p.counters;
  int* const exits = p.counters + 1;
  int* const done = p.counters + 2;

  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(full0 + 8 * s, 1);      // used on the leader: its own arrive + both CTAs' bytes
      mbar_init(empty0 + 8 * s, 1);     // one commit from the leader's MMA thread, in each CTA
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(tfull0 + 8 * a, 1);
      mbar_init(tempty0 + 8 * a, 2 * kEpiWarps);    // used on the leader: the epilogue warps of both CTAs
    }
    for (int i = 0; i < kRing; ++i) {
      mbar_init(rfull0 + 8 * i, 1);     // the leader's producer, in each CTA
      // used on the leader: its MMA issuer, the partner's producer, the epilogue warps of both CTAs
      mbar_init(rempty0 + 8 * i, 2 + 2 * kEpiWarps);
    }
    *abort_flag = 0;
    fence_barrier_init();
    fence_proxy_async_smem();
  }
  if (warp == 1) {
    tmem_alloc_pair(smem_u32(tmem_slot), 2 * kPairBN);
    tmem_relinquish_pair();
  }
  for (int i = threadIdx.x; i < p.n_ops; i += kChainThreads) build_op(ops[i], p.ops[i], p);
  for (int i = threadIdx.x; i < p.n_maps; i += kChainThreads) tma_prefetch_desc(p.maps + i);
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();                    // both CTAs' barriers exist before anything crosses the pair
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  int fail_code = 0;

  if (warp == 0) {
    if (lane == 0) {
      // ---------------- tickets (leader) and TMA (both CTAs) ----------------
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      int t = leader ? atomicAdd(ticket, 1) : 0;
      for (uint32_t cnt = 0; ok; ++cnt) {
        const uint32_t slot = cnt % kRing;
        const uint32_t turn = (cnt / kRing) & 1u;
        int4 e;
        if (leader) {
          if (!mbar_wait_cluster_bounded(rempty0 + 8 * slot, turn ^ 1u, abort_flag)) {
            fail_code = kStatusTimeoutProducer;
            break;
          }
          e = make_int4(-1, 0, 0, 0);
          if (t < p.total) e = __ldg(p.tab + t);
          ring[slot] = e;
          mbar_arrive(rfull0 + 8 * slot);
          st_cluster_v4(mapa_shared(smem_u32(ring + slot), 1), e);
          mbar_arrive_cluster(mapa_shared(rfull0 + 8 * slot, 1));
          if (e.x < 0) break;
        } else {
          if (!mbar_wait_cluster_bounded(rfull0 + 8 * slot, turn, abort_flag)) {
            fail_code = kStatusTimeoutProducer;
            break;
          }
          e = ring[slot];
          mbar_arrive_cluster(mapa_shared(rempty0 + 8 * slot, 0));
          if (e.x < 0) break;
        }
        const OpS& op = ops[entry_op(e)];
        if (e.w > 0) {
          if (!wait_count(done + entry_ctr(e), e.w, abort_flag)) {
            fail_code = kStatusTimeoutChain;
            break;
          }
          fence_proxy_async_global();      // other CTAs' stores before this thread's bulk loads
        }
        if (leader) t = atomicAdd(ticket, 1);    // once this tile can run, see above
        const CUtensorMap* tmA = p.maps + op.map_a;
        const CUtensorMap* tmB = p.maps + op.map_b;
        const int halves = entry_halves<WIDE>(e);
        const int m0 = entry_m(e) * 256 + 128 * static_cast<int>(rank);
        const int n0 = entry_n(e) * kPairBN + 128 * static_cast<int>(rank);
        const int b = entry_b(e);
        const int a_mn = op.k.a_mn_major, b_mn = op.k.b_mn_major;
        const int num_kb = (op.k.K + BK - 1) / BK;
        const uint32_t bytes = 2 * (C::kABytes + halves * C::kBBytes);    // of both CTAs
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!mbar_wait_bounded(empty0 + 8 * stage, phase ^ 1u, abort_flag)) {
            ok = false;
            fail_code = kStatusTimeoutProducer;
            break;
          }
          if (leader) mbar_arrive_expect_tx(full0 + 8 * stage, bytes);
          const uint32_t fb = (full0 + 8 * stage) & 0xFEFFFFFFu;     // the leader's barrier
          const uint32_t a_dst = smem_u32(sA + stage * C::kABytes);
          if (!a_mn) {
            tma_load_3d_pair(a_dst, tmA, fb, kb * BK, m0, b);
          } else {
#pragma unroll
            for (int mb = 0; mb < 2; ++mb)
              tma_load_3d_pair(a_dst + mb * kBlockBytes, tmA, fb, m0 + 64 * mb, kb * BK, b);
          }
          for (int h = 0; h < halves; ++h) {
            const uint32_t b_dst = smem_u32(sB + (C::kHalves * stage + h) * C::kBBytes);
            const int n = n0 + h * kPairBN;
            if (!b_mn) {
              tma_load_3d_pair(b_dst, tmB, fb, kb * BK, n, b);
            } else {
#pragma unroll
              for (int nb = 0; nb < 2; ++nb)
                tma_load_3d_pair(b_dst + nb * kBlockBytes, tmB, fb, n + 64 * nb, kb * BK, b);
            }
          }
          if (++stage == S) {
            stage = 0;
            phase ^= 1u;
          }
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0 && leader) {
      // ---------------- MMA issuer (leader only) ----------------
      uint32_t it = 0;                     // k-blocks consumed so far: stage it % S, trip it / S
      int acc = 0;
      uint32_t acc_phase = 0;              // one bit per accumulator
      for (uint32_t cnt = 0;; ++cnt) {
        const uint32_t slot = cnt % kRing;
        if (!mbar_wait_bounded(rfull0 + 8 * slot, (cnt / kRing) & 1u, abort_flag)) {
          fail_code = kStatusTimeoutMma;
          break;
        }
        const int4 e = ring[slot];
        mbar_arrive(rempty0 + 8 * slot);
        if (e.x < 0) break;
        const OpS& op = ops[entry_op(e)];
        const int a_mn = op.k.a_mn_major, b_mn = op.k.b_mn_major;
        const uint32_t idesc = make_idesc_f16(256, kPairBN, op.k.ab_fp16 != 0, a_mn != 0, b_mn != 0);
        const int num_kb = (op.k.K + BK - 1) / BK;
        const int halves = entry_halves<WIDE>(e);

        auto wait_acc = [&](int a) -> bool {          // accumulator `a` has been drained
          const bool r = mbar_wait_bounded(tempty0 + 8 * a, ((acc_phase >> a) & 1u) ^ 1u, abort_flag);
          acc_phase ^= 1u << a;
          tc_fence_after_sync();
          return r;
        };
        auto wait_full = [&](int kb) -> bool {
          const uint32_t i = it + kb;
          const bool r = mbar_wait_bounded(full0 + 8 * (i % S), (i / S) & 1u, abort_flag);
          tc_fence_after_sync();
          return r;
        };
        auto mma = [&](int a, int h, int kb) {        // one k-block of half h into accumulator a
          const uint32_t st = (it + kb) % S;
          const uint32_t a_base = smem_u32(sA + st * C::kABytes);
          const uint32_t b_base = smem_u32(sB + (C::kHalves * st + h) * C::kBBytes);
          const uint32_t d_tmem = tmem_base + static_cast<uint32_t>(a * kPairBN);
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k) {
            const uint64_t adesc = a_mn ? make_smem_desc_sw128(a_base + k * 2048, kBlockBytes, 1024)
                                        : make_smem_desc_sw128(a_base + k * 32, 16, 1024);
            const uint64_t bdesc = b_mn ? make_smem_desc_sw128(b_base + k * 2048, kBlockBytes, 1024)
                                        : make_smem_desc_sw128(b_base + k * 32, 16, 1024);
            umma_f16_ss_pair(d_tmem, adesc, bdesc, idesc, (kb | k) != 0 ? 1u : 0u);
          }
        };
        auto commit = [&](uint32_t bar) {             // the MMAs so far, in both CTAs
          umma_commit_pair(mapa_shared(bar, 0));
          umma_commit_pair(mapa_shared(bar, 1));
        };

        bool ok = wait_acc(acc);
        if (halves == 1) {
          for (int kb = 0; ok && kb < num_kb; ++kb) {
            ok = wait_full(kb);
            if (!ok) break;
            mma(acc, 0, kb);
            commit(empty0 + 8 * ((it + kb) % S));
          }
          if (ok) commit(tfull0 + 8 * acc);
          acc ^= 1;
        } else {
          // k-blocks [0, head) and [tail, num_kb) half by half, those between together
          const int head = min(S, num_kb);
          const int tail = max(head, num_kb - S);
          for (int kb = 0; ok && kb < head; ++kb) {
            ok = wait_full(kb);
            if (ok) mma(acc, 0, kb);
          }
          if (ok && head == num_kb) commit(tfull0 + 8 * acc);
          ok = ok && wait_acc(acc ^ 1);
          for (int kb = 0; ok && kb < head; ++kb) {
            mma(acc ^ 1, 1, kb);
            commit(empty0 + 8 * ((it + kb) % S));
          }
          for (int kb = head; ok && kb < tail; ++kb) {
            ok = wait_full(kb);
            if (!ok) break;
            mma(acc, 0, kb);
            mma(acc ^ 1, 1, kb);
            commit(empty0 + 8 * ((it + kb) % S));
          }
          for (int kb = tail; ok && kb < num_kb; ++kb) {
            ok = wait_full(kb);
            if (ok) mma(acc, 0, kb);
          }
          if (ok && head < num_kb) commit(tfull0 + 8 * acc);
          for (int kb = tail; ok && kb < num_kb; ++kb) {
            mma(acc ^ 1, 1, kb);
            commit(empty0 + 8 * ((it + kb) % S));
          }
          if (ok) commit(tfull0 + 8 * (acc ^ 1));
        }
        if (!ok) {
          fail_code = kStatusTimeoutMma;
          break;
        }
        it += num_kb;
      }
    }
  } else {
    // ---------------- epilogue (warps 2..9 of both CTAs) ----------------
    const int q = warp & 3;              // TMEM lane quarter this warp may read
    const int part = (warp - 2) >> 2;    // which 128 of a half's 256 columns
    uint8_t* const stage_mem = staging + (warp - 2) * kStageWarpBytes;
    int acc = 0;
    uint32_t acc_phase = 0;              // one bit per accumulator
    bool ok = true;
    for (uint32_t cnt = 0; ok; ++cnt) {
      const uint32_t slot = cnt % kRing;
      if (!__all_sync(0xffffffffu, mbar_wait_cluster_bounded(rfull0 + 8 * slot, (cnt / kRing) & 1u, abort_flag))) {
        fail_code = kStatusTimeoutEpilogue;
        break;
      }
      const int4 e = ring[slot];
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(mapa_shared(rempty0 + 8 * slot, 0));
      if (e.x < 0) break;
      const OpS& op = ops[entry_op(e)];
      const int halves = entry_halves<WIDE>(e);
      for (int h = 0; h < halves; ++h) {
        const TileEpilogue tile(op.k, entry_b(e), entry_m(e) * 256 + 128 * static_cast<int>(rank) + q * 32,
                                entry_mirror_half(e, h), stage_mem, lane);
        bool ready = true;
        if (lane == 0 && e.w > 0 && tile.add_c) {
          // C was stored by other CTAs: one lane acquires for the warp, the reads go to L2
          ready = wait_count(done + entry_ctr(e), e.w, abort_flag);
          if (!ready) fail_code = kStatusTimeoutChain;
        }
        ok = __all_sync(0xffffffffu, ready);
        if (!ok) break;
        const int col0 = (entry_n(e) + h) * kPairBN + part * (kPairBN / 2);
        RawC c;
        tile.fetch_c(c, col0);           // arrives while the product runs
        ready = mbar_wait_bounded(tfull0 + 8 * acc, (acc_phase >> acc) & 1u, abort_flag);
        if (!ready) fail_code = kStatusTimeoutEpilogue;
        ok = __all_sync(0xffffffffu, ready);
        if (!ok) break;
        tc_fence_after_sync();
        tile.run(tmem_base + (static_cast<uint32_t>(q * 32) << 16) +
                     static_cast<uint32_t>(acc * kPairBN + part * (kPairBN / 2)),
                 col0, kPairBN / 2, c);
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) {
          mbar_arrive_cluster(mapa_shared(tempty0 + 8 * acc, 0));   // the leader's barrier
          red_add_release_gpu(done + entry_ctr(e), 1);              // covers the stores of the whole warp
        }
        acc_phase ^= 1u << acc;
        acc ^= 1;
      }
    }
  }

  // ---------------- teardown ----------------
  tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag) {
    if (fail_code != 0 && p.status != nullptr) atomicCAS(p.status, 0, fail_code);
    // bulk copies that may still be in flight land before the shared memory is handed on
    for (int i = 0; i < 64; ++i) __nanosleep(2000);
    __syncthreads();
  }
  cluster_sync_all();                    // the peer may still read or signal this CTA's shared memory until here
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc_pair(tmem_base, 2 * kPairBN);
  }
  if (warp == 0) {
    int last = 0;
    if (lane == 0) {
      __threadfence();
      last = atomicAdd(exits, 1) == static_cast<int>(gridDim.x) - 1;
    }
    if (__shfl_sync(0xffffffffu, last, 0)) {
      for (int i = lane; i < p.n_counters; i += 32) p.counters[i] = 0;
    }
  }
}

ChainParams make_params(const DmuonChainArgs& a) {
  ChainParams p;
  memcpy(p.maps, a.maps, static_cast<size_t>(a.n_maps) * sizeof(CUtensorMap));
  p.ops = static_cast<const DmuonChainOp*>(a.ops);
  p.tab = reinterpret_cast<const int4*>(a.tab);
  p.counters = a.counters;
  p.work = static_cast<char*>(a.work);
  p.status = a.status;
  p.n_ops = a.n_ops; p.n_maps = a.n_maps; p.total = a.total; p.n_counters = a.n_counters;
  for (int i = 0; i < DMUON_CHAIN_MAX_GROUPS; ++i) p.fin[i] = a.fin[i];
  return p;
}

template <bool WIDE>
int launch_chain_pair(const DmuonChainArgs& a, cudaStream_t stream, int sms) {
  cudaError_t err = cudaFuncSetAttribute(chain_pair_kernel<WIDE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         pair_smem_bytes<WIDE>(DMUON_CHAIN_MAX_OPS));
  if (err != cudaSuccess) return static_cast<int>(err);
  int pairs = sms / 2;
  if (a.total < pairs) pairs = a.total;
  if (pairs < 1) pairs = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * pairs, 1, 1);
  cfg.blockDim = dim3(kChainThreads, 1, 1);
  cfg.dynamicSmemBytes = pair_smem_bytes<WIDE>(a.n_ops);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  err = cudaLaunchKernelEx(&cfg, chain_pair_kernel<WIDE>, make_params(a));
  count_launch();
  return static_cast<int>(err != cudaSuccess ? err : cudaGetLastError());
}

template <int BN>
int launch_chain(const DmuonChainArgs& a, cudaStream_t stream, int sms) {
  auto kern = chain_kernel<BN>;
  const int bytes = chain_smem_bytes<BN>(a.n_ops);
  cudaError_t err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         chain_smem_bytes<BN>(DMUON_CHAIN_MAX_OPS));
  if (err != cudaSuccess) return static_cast<int>(err);
  const int grid = a.total < sms ? a.total : sms;
  kern<<<grid, kChainThreads, bytes, stream>>>(make_params(a));
  count_launch();
  return static_cast<int>(cudaGetLastError());
}

}  // namespace
}  // namespace dmuon

extern "C" int dmuon_chain_encode_maps(const DmuonChainMap* maps, int n, void* out_host) {
  CUtensorMap* out = static_cast<CUtensorMap*>(out_host);
  if ((reinterpret_cast<uintptr_t>(out) & 63) != 0) return -1;
  for (int i = 0; i < n; ++i) {
    const DmuonChainMap& m = maps[i];
    if ((m.ld % 8) != 0 || (m.batch_stride % 8) != 0 || (reinterpret_cast<uintptr_t>(m.base) & 15)) return -1;
    const int rc = dmuon::make_map(out + i, m.base, m.fp16 != 0, m.cols, m.rows, m.batch, m.ld, m.batch_stride,
                                   m.box_cols, m.box_rows);
    if (rc != 0) return rc;
  }
  return 0;
}

extern "C" int dmuon_chain_launch(const DmuonChainArgs* args, void* stream_v) {
  using namespace dmuon;
  const DmuonChainArgs& a = *args;
  if (a.total <= 0) return 0;
  if (a.n_ops <= 0 || a.n_ops > DMUON_CHAIN_MAX_OPS || a.n_final < 0 || a.n_final > DMUON_CHAIN_MAX_GROUPS) return -1;
  if (a.n_maps <= 0 || a.n_maps > DMUON_CHAIN_MAX_MAPS) return -1;
  if (a.ops == nullptr || a.maps == nullptr || a.tab == nullptr || a.counters == nullptr || a.work == nullptr) return -1;
  for (int i = 0; i < a.n_final; ++i) {
    const DmuonChainFinal& f = a.fin[i];
    if ((reinterpret_cast<uintptr_t>(f.D) & 15) || (reinterpret_cast<uintptr_t>(f.C) & 15)) return -1;
    if ((f.ldc % 8) || (f.ldd % 8) || (f.ldd2 % 8) || (f.strideC % 8) || (f.strideD % 8)) return -1;
  }
  int dev = 0, sms = 0;
  cudaError_t err = cudaGetDevice(&dev);
  if (err == cudaSuccess) err = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (err != cudaSuccess) return static_cast<int>(err);
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_v);
  if (a.bn == 64) return launch_chain<64>(a, stream, sms);
  if (a.bn == 128) return launch_chain<128>(a, stream, sms);
  if (a.bn == 256) return a.wide ? launch_chain_pair<true>(a, stream, sms) : launch_chain_pair<false>(a, stream, sms);
  return -1;
}
