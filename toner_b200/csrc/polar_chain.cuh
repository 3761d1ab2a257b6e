// All products of a Newton-Schulz polar iteration in one launch.
//
// Per step and matrix: Gram, polynomial, update (toner_ns_polar).  Launched one by one, products of a few waves of short tiles
// spend a good part of their time on their first copies, on their last tiles' results -- 10000 to 14000 cycles, where the MMAs of
// depth 768 take 6500 -- and on the hand-over.  Here the CTAs (pairs) take tiles of all products in their order from a counter; a
// tile waits only for the tiles of the previous product on ITS matrix, so one matrix's products overlap another's.  Ten steps, launched
// / chained, us: 32 x 768^2 1173 / 976, 12 x 768^2 586 / 462, 4 x 768^2 341 / 287, 8 x 3072 x 768 952 / 872, 16 x 1280^2
// 1816 / 1592; 768^2 alone 254 / 254.  What bounds it then is the SM's way to L2: a 256 x 256 tile of an update moves 704 KB
// a CTA, at 42 bytes a cycle.
//
// A unit is one tile of one product; the order is steps, then Gram / polynomial / update, then matrices, then tiles.  done[b]
// counts the CTAs that have finished their part of a tile of matrix b; a unit of a product needs every tile of the products
// before it on b (which also orders every buffer's reuse).  A unit's needs precede it in the order, and units are claimed in order
// by CTAs that are running and process their claims in order, so the earliest unfinished unit can always proceed, whatever
// other kernels hold of the GPU.  Every wait is bounded all the same.
#pragma once

#include "gemm_tcgen05.cuh"

namespace toner {

struct PolarChain {
  GemmParams op[6];      // Gram of x0 / x1, polynomial, update x0 -> x1 / x1 -> x0, last update
  int steps, batch;
  int tiles[3];          // per matrix: Gram, polynomial, update
  unsigned int* claim;   // next unit (zeroed before the launch, as done[batch] is)
  unsigned int* done;
};

// What a tile waits for and what it reports costs thousands of cycles under load (an acquire 6000, a release 3000), so neither
// is done by the threads that copy, multiply or write: two warps of their own follow the claims, one a few units ahead until
// what a unit needs is there, one behind until all of its results are.
constexpr int kClaims = 3;           // units in flight per CTA (pair)
constexpr int kChainThreads = 512;   // copies, MMAs, claims | needs, reports | epilogue (two warpgroups)

template <int BN, bool kPair>
__global__ void __launch_bounds__(kChainThreads, 1) polar_chain_kernel(const __grid_constant__ PolarChain c) {
  using S = GemmSmem<BN, kPair>;
  static_assert(BN <= 256, "double-buffered accumulators");
  constexpr int TM = kPair ? 2 * kBM : kBM;
  constexpr int kCtas = kPair ? 2 : 1;
  constexpr unsigned kArrivals = kCtas;   // reports a tile makes
  const uint32_t cta_rank = kPair ? ptx::cluster_ctarank() : 0u;
  const bool leader = cta_rank == 0;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = ptx::smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t* const smem = smem_raw + (base - raw);
  const uint32_t bars = base + S::kTileBytes + S::kEpiBytes;
  auto full_bar = [&](int s) { return bars + 8u * s; };
  auto empty_bar = [&](int s) { return bars + 8u * (S::kStages + s); };
  auto tfull_bar = [&](int s) { return bars + 8u * (2 * S::kStages + s); };
  auto tempty_bar = [&](int s) { return bars + 8u * (2 * S::kStages + 2 + s); };
  auto c_bar = [&](int w) { return bars + 8u * (2 * S::kStages + 4 + w); };
  auto claimed_bar = [&](int s) { return bars + 8u * (2 * S::kStages + 12 + s); };                // a unit's number is there
  auto taken_bar = [&](int s) { return bars + 8u * (2 * S::kStages + 12 + kClaims + s); };        // every role is done with it (leader's)
  auto ready_bar = [&](int s) { return bars + 8u * (2 * S::kStages + 12 + 2 * kClaims + s); };    // what the unit needs is there
  auto written_bar = [&](int s) { return bars + 8u * (2 * S::kStages + 12 + 3 * kClaims + s); };  // its results are
  constexpr int kBars = 2 * S::kStages + 12 + 4 * kClaims;
  constexpr int kAfterBars = S::kTileBytes + S::kEpiBytes + 8 * kBars;
  static_assert(8 * kBars + 8 + 4 * kClaims <= S::kBarBytes, "barrier block");
  volatile uint32_t* const tmem_slot = reinterpret_cast<volatile uint32_t*>(smem + kAfterBars);
  volatile int* const abort_flag = reinterpret_cast<volatile int*>(smem + kAfterBars + 4);
  volatile uint32_t* const claims = reinterpret_cast<volatile uint32_t*>(smem + kAfterBars + 8);
  int* const status = c.op[0].status;
  auto raise_abort = [&]() {
    *abort_flag = 1;
    if constexpr (kPair)
      ptx::st_cluster_u32(ptx::mapa(ptx::smem_u32(const_cast<int*>(abort_flag)), cta_rank ^ 1u), 1u);
  };

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned step_tiles = c.tiles[0] + c.tiles[1] + c.tiles[2];
  const unsigned units = step_tiles * c.batch * c.steps;
  struct Work {
    int op, b, tile, tiles;
    unsigned need;   // reports at done[b] before this unit may start
  };
  auto work_of = [&](unsigned u) {
    const unsigned per = step_tiles * c.batch, step = u / per;
    unsigned r = u - step * per, before = 0;
    int kind = 0;
    while (kind < 2 && r >= (unsigned)(c.tiles[kind] * c.batch)) {
      r -= c.tiles[kind] * c.batch;
      before += c.tiles[kind];
      ++kind;
    }
    Work w;
    w.tiles = c.tiles[kind];
    w.b = (int)(r / w.tiles);
    w.tile = (int)r - w.b * w.tiles;
    w.op = kind == 0 ? (int)(step & 1) : (kind == 1 ? 2 : (step + 1 == (unsigned)c.steps ? 5 : 3 + (int)(step & 1)));
    w.need = kArrivals * (step * step_tiles + before);
    return w;
  };

  if (threadIdx.x == 0) {
    for (int s = 0; s < S::kStages; ++s) {
      ptx::mbar_init(full_bar(s), 1);
      ptx::mbar_init(empty_bar(s), 1);
    }
    for (int s = 0; s < 2; ++s) {
      ptx::mbar_init(tfull_bar(s), 1);
      ptx::mbar_init(tempty_bar(s), 8 * kCtas);
    }
    for (int w = 0; w < 8; ++w) ptx::mbar_init(c_bar(w), 1);
    for (int s = 0; s < kClaims; ++s) {
      ptx::mbar_init(claimed_bar(s), 1);
      ptx::mbar_init(taken_bar(s), 12 * kCtas + 1);   // a CTA's two producers, needs, reports, eight epilogue warps; the MMA issuer
      ptx::mbar_init(ready_bar(s), 1);
      ptx::mbar_init(written_bar(s), 8);
    }
    *abort_flag = 0;
    ptx::fence_mbar_init();
  }
  if (warp == 1) {
    if constexpr (kPair) {
      ptx::tmem_alloc_pair(ptx::smem_u32(const_cast<uint32_t*>(tmem_slot)), S::kTmemCols);
      ptx::tmem_relinquish_pair();
    } else {
      ptx::tmem_alloc(ptx::smem_u32(const_cast<uint32_t*>(tmem_slot)), S::kTmemCols);
      ptx::tmem_relinquish();
    }
  }
  ptx::tc_fence_before();
  if constexpr (kPair) ptx::cluster_sync();
  else __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  ptx::pdl_begin();

  // A role's view of the claims: the next unit of this CTA (pair), `units` once there is none, ~0 after an abort.
  int turn = 0;
  uint32_t turn_parity = 0;
  auto await_claim = [&]() {
    return ptx::mbar_wait_unless<true>(claimed_bar(turn), turn_parity, kWaitCycles, abort_flag) ? claims[turn] : ~0u;
  };
  auto claim_read = [&]() {   // (one thread of the role; it needs the slot's barriers no more)
    if constexpr (kPair) ptx::mbar_arrive_cluster_release(ptx::mapa(taken_bar(turn), 0));
    else ptx::mbar_arrive(taken_bar(turn));
  };
  auto next_turn = [&]() {
    if (++turn == kClaims) {
      turn = 0;
      turn_parity ^= 1u;
    }
  };
  // the claimed unit's needs are met (the warp that looks after them says so)
  auto await_ready = [&]() { return ptx::mbar_wait_unless(ready_bar(turn), turn_parity, kWaitCycles, abort_flag); };

  if (warp < 4) {
    if (warp == 3) {
      // ---------------------------------------------------------- claims units, for both CTAs of a pair
      if (leader && ptx::elect_one()) {
        for (;;) {
          if (!ptx::mbar_wait_unless<true>(taken_bar(turn), turn_parity ^ 1u, kWaitCycles, abort_flag)) {
            report(status, kTimeoutProducer);
            raise_abort();
            break;
          }
          const uint32_t u = min(atomicAdd(c.claim, 1u), units);
          claims[turn] = u;
          ptx::mbar_arrive(claimed_bar(turn));
          if constexpr (kPair) {
            ptx::st_cluster_u32(ptx::mapa(ptx::smem_u32(const_cast<uint32_t*>(claims + turn)), 1), u);
            ptx::mbar_arrive_cluster_release(ptx::mapa(claimed_bar(turn), 1));
          }
          if (u == units) break;
          next_turn();
        }
      }
    } else if (warp == 0 || warp == 2) {
      // ---------------------------------------------------------- TMA producers: warp 0 brings A, warp 2 brings B
      const bool for_a = warp == 0;
      if (ptx::elect_one()) {
        int stage = 0;
        uint32_t phase = 0;
        bool ok = true;
        while (ok) {
          const uint32_t u = await_claim();
          if (u == ~0u) ok = false;
          if (u >= units) break;
          const Work w = work_of(u);
          const GemmParams& p = c.op[w.op];
          const bool ready = await_ready();
          claim_read();
          next_turn();
          if (!ready) {
            report(status, kTimeoutProducer);
            raise_abort();
            ok = false;
            break;
          }
          int b, tm, tn;
          tile_coord(p, BN, TM, w.tile, w.tiles, (p.N + BN - 1) / BN, b, tm, tn);
          const CUtensorMap* const map = for_a ? &p.a_map : &p.b_map;
          const int mn = for_a ? p.a_mn : p.b_mn;
          const int first = for_a ? tm * TM + (int)cta_rank * kBM : tn * BN + (int)cta_rank * S::kBRows;
          const int rows = for_a ? kBM : S::kBRows;
          const int num_kb = (p.K + kBK - 1) / kBK;
          for (int kb = 0; kb < num_kb; ++kb) {
            if (!ptx::mbar_wait_unless(empty_bar(stage), phase ^ 1u, kWaitCycles, abort_flag)) {
              report(status, kTimeoutProducer);
              raise_abort();
              ok = false;
              break;
            }
            const uint32_t dst = base + stage * S::kStageBytes + (for_a ? 0 : S::kABytes);
            if constexpr (kPair) {
              const uint32_t lbar = ptx::mapa(full_bar(stage), 0);
              if (for_a && leader) ptx::mbar_expect_tx(full_bar(stage), 2 * S::kStageBytes);
              if (mn) {
                for (int s = 0; s < rows / 64; ++s) ptx::tma_load_3d_pair(dst + s * 8192, map, lbar, first + s * 64, kb * kBK, w.b);
              } else {
                ptx::tma_load_3d_pair(dst, map, lbar, kb * kBK, first, w.b);
              }
            } else {
              if (for_a) ptx::mbar_expect_tx(full_bar(stage), S::kStageBytes);
              if (mn) {
                for (int s = 0; s < rows / 64; ++s) ptx::tma_load_3d(dst + s * 8192, map, full_bar(stage), first + s * 64, kb * kBK, w.b);
              } else {
                ptx::tma_load_3d(dst, map, full_bar(stage), kb * kBK, first, w.b);
              }
            }
            if (++stage == S::kStages) {
              stage = 0;
              phase ^= 1u;
            }
          }
        }
        if (!ok || *abort_flag) {   // (as in gemm_tcgen05_kernel: copies already issued must land before the CTA ends)
          if (!kPair || leader) {
            for (int s = 0; s < S::kStages; ++s)
              ptx::mbar_wait(full_bar(s), (s < stage) ? phase : (phase ^ 1u), kDrainCycles);
          }
          const long long t0 = clock64();
          while (clock64() - t0 < kSettleCycles) {
          }
        }
      }
    } else {
      // ---------------------------------------------------------- MMA issuer (of a pair: the leader CTA only)
      if (leader && ptx::elect_one()) {
        const uint32_t desc_hi = (1024u >> 4) | (1u << 14) | (2u << 29);
        int stage = 0;
        uint32_t phase = 0, tile = 0;
        bool ok = true;
        auto gave_up = [&]() {
          report(status, kTimeoutMma);
          raise_abort();
          ok = false;
        };
        while (ok) {
          const uint32_t u = await_claim();
          if (u >= units) break;   // (~0 as well)
          claim_read();
          next_turn();
          const GemmParams& p = c.op[work_of(u).op];
          const uint32_t idesc = (1u << 4) | ((uint32_t)p.fmt << 7) | ((uint32_t)p.fmt << 10) | ((uint32_t)p.a_mn << 15) |
                                 ((uint32_t)p.b_mn << 16) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(TM >> 4) << 24);
          const uint32_t a_const = ((p.a_mn ? 8192u : 16u) >> 4) << 16, b_const = ((p.b_mn ? 8192u : 16u) >> 4) << 16;
          const uint32_t a_step = (p.a_mn ? 2048u : 32u) >> 4, b_step = (p.b_mn ? 2048u : 32u) >> 4;
          const int num_kb = (p.K + kBK - 1) / kBK;
          const int buf = (int)(tile & 1u);
          if (!ptx::mbar_wait_unless(tempty_bar(buf), ((tile >> 1) & 1u) ^ 1u, kWaitCycles, abort_flag)) {
            gave_up();
            break;
          }
          ptx::tc_fence_after();
          const uint32_t d_tmem = tmem_base + (uint32_t)(buf * BN);
          for (int kb = 0; kb < num_kb && ok; ++kb) {
            if (!ptx::mbar_wait_unless(full_bar(stage), phase, kWaitCycles, abort_flag)) {
              gave_up();
              break;
            }
            ptx::tc_fence_after();
            const uint32_t at = base + stage * S::kStageBytes;
            const uint32_t a_lo = ((at & 0x3FFFFu) >> 4) | a_const, b_lo = (((at + S::kABytes) & 0x3FFFFu) >> 4) | b_const;
#pragma unroll
            for (int k = 0; k < kBK / kUmmaK; ++k) {
              const uint64_t da = ((uint64_t)desc_hi << 32) | (a_lo + k * a_step), db = ((uint64_t)desc_hi << 32) | (b_lo + k * b_step);
              const uint32_t more = (kb | k) != 0 ? 1u : 0u;
              if constexpr (kPair) ptx::mma_f16_pair(d_tmem, da, db, idesc, more);
              else ptx::mma_f16(d_tmem, da, db, idesc, more);
            }
            if constexpr (kPair) {
              ptx::mma_commit_pair(empty_bar(stage));
              ptx::mma_commit_pair(ptx::mapa(empty_bar(stage), 1));
            } else {
              ptx::mma_commit(empty_bar(stage));
            }
            if (++stage == S::kStages) {
              stage = 0;
              phase ^= 1u;
            }
          }
          if (ok) {
            if constexpr (kPair) {
              ptx::mma_commit_pair(tfull_bar(buf));
              ptx::mma_commit_pair(ptx::mapa(tfull_bar(buf), 1));
            } else {
              ptx::mma_commit(tfull_bar(buf));
            }
          }
          ++tile;
        }
      }
    }
  } else if (warp < 8) {
    if (warp == 4) {
      // ---------------------------------------------------------- needs: done[b] has counted every tile the unit waits for
      if (ptx::elect_one()) {
        for (;;) {
          const uint32_t u = await_claim();
          if (u >= units) break;
          const Work w = work_of(u);
          if (w.need) {
            const long long t0 = clock64();
            bool there = ptx::ld_acquire_gpu(c.done + w.b) >= w.need;
            while (!there && !*abort_flag && clock64() - t0 < kWaitCycles) {
              __nanosleep(32);
              there = ptx::ld_acquire_gpu(c.done + w.b) >= w.need;
            }
            if (!there) {
              report(status, kTimeoutProducer);
              raise_abort();
              break;
            }
            ptx::fence_proxy_async();   // the copies that follow read what was written there by copies
          }
          ptx::mbar_arrive(ready_bar(turn));
          claim_read();
          next_turn();
        }
      }
    } else if (warp == 5) {
      // ---------------------------------------------------------- reports: every store of this CTA's part has been made
      if (ptx::elect_one()) {
        for (;;) {
          const uint32_t u = await_claim();
          if (u >= units) break;
          if (!ptx::mbar_wait_unless(written_bar(turn), turn_parity, kWaitCycles, abort_flag)) {
            report(status, kTimeoutEpilogue);
            raise_abort();
            break;
          }
          ptx::red_release_gpu(c.done + work_of(u).b, 1u);
          claim_read();   // (only now: a slot's barriers are used again when every role is done with its unit)
          next_turn();
        }
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue (warps 8..15), as in gemm_tcgen05_kernel
    constexpr int NCH = BN / 64;
    const int lane_group = warp & 3, half = (warp - 8) >> 2, ew = warp - 8;
    const uint32_t warp_bufs = base + S::kTileBytes + ew * S::kEpiBufs * kEpiBlockBytes;
    EpilogueRing ring{warp_bufs, S::kEpiBufs};
    static_assert(S::kEpiBufs == 2, "C has the second block where there is C");
    uint32_t c_buf = 0, c_phase = 0, tile = 0;
    bool alive = true;
    auto gave_up = [&]() {
      if (lane == 0) {
        report(status, kTimeoutEpilogue);
        raise_abort();
      }
      alive = false;
    };
    while (alive) {
      const uint32_t u = await_claim();
      if (!__all_sync(0xffffffffu, u < units ? 1 : 0)) break;
      const uint32_t written = written_bar(turn);
      const Work w = work_of(u);
      const GemmParams& p = c.op[w.op];
      const int b = w.b;
      int unused, tm, tn;
      tile_coord(p, BN, TM, w.tile, w.tiles, (p.N + BN - 1) / BN, unused, tm, tn);
      const int row_first = tm * TM + (int)cta_rank * kBM + lane_group * 32;
      const int col_first = tn * BN + half * (BN / 2);
      auto needed = [&](int c0) { return c0 < p.N && row_first < p.M && !(p.tri && c0 + 31 < row_first); };
      const int buf = (int)(tile & 1u);
      EpilogueTile e;
      e.alpha = p.alpha;
      e.beta = p.beta;
      e.use_c = p.C != nullptr;
      e.stats = p.maxabs != nullptr;
      int cc_first = 0, cc_end = NCH;
      while (cc_first < NCH && !needed(col_first + cc_first * 32)) ++cc_first;
      while (cc_end > cc_first && !needed(col_first + (cc_end - 1) * 32)) --cc_end;
      // C has a block of its own; results then leave from the other.  (Both are free: a tile ends with all of its stores made.)
      ring = EpilogueRing{warp_bufs, e.use_c ? 1 : 2};
      auto fetch_c = [&](int cc) {
        if (!e.use_c || cc >= cc_end) return;
        c_buf = warp_bufs + kEpiBlockBytes;
        if (ptx::elect_one()) {
          ptx::mbar_expect_tx(c_bar(ew), kEpiBlockBytes);
          ptx::tma_load_3d(c_buf, &p.c_map, c_bar(ew), col_first + cc * 32, row_first, b);
        }
      };
      if (e.use_c && cc_first < cc_end) {
        if (!__all_sync(0xffffffffu, await_ready() ? 1 : 0)) {
          gave_up();
          break;
        }
        fetch_c(cc_first);
      }
      __syncwarp();
      if (ptx::elect_one()) claim_read();
      next_turn();
      if (!__all_sync(0xffffffffu, ptx::mbar_wait_unless(tfull_bar(buf), (tile >> 1) & 1u, kWaitCycles, abort_flag) ? 1 : 0)) {
        gave_up();
        break;
      }
      ptx::tc_fence_after();
      auto release = [&]() {
        ptx::tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          if constexpr (kPair) ptx::mbar_arrive_cluster(ptx::mapa(tempty_bar(buf), 0));
          else ptx::mbar_arrive(tempty_bar(buf));
        }
      };
      EpilogueSums sums;
      const uint32_t taddr = tmem_base + ((uint32_t)(lane_group * 32) << 16) + (uint32_t)(buf * BN + half * (BN / 2));
#pragma unroll 1
      for (int cc = cc_first; cc < cc_end; ++cc) {
        const int c0 = col_first + cc * 32;
        float v[32];
        {
          uint32_t r[32];
          ptx::tmem_ld32(taddr + (uint32_t)(cc * 32), r);
          ptx::tmem_ld_wait();
          if (cc == cc_end - 1) release();
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
        }
        if (e.use_c) {
          if (!__all_sync(0xffffffffu, ptx::mbar_wait_unless(c_bar(ew), c_phase, kWaitCycles, abort_flag) ? 1 : 0)) {
            gave_up();
            break;
          }
          float4 r[8];
          load_row_f32(c_buf, lane, r);
          c_buf = 0;
          c_phase ^= 1u;
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            v[4 * j] = fmaf(e.beta, r[j].x, e.alpha * v[4 * j]);
            v[4 * j + 1] = fmaf(e.beta, r[j].y, e.alpha * v[4 * j + 1]);
            v[4 * j + 2] = fmaf(e.beta, r[j].z, e.alpha * v[4 * j + 2]);
            v[4 * j + 3] = fmaf(e.beta, r[j].w, e.alpha * v[4 * j + 3]);
          }
          __syncwarp();
          fetch_c(cc + 1);
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] *= e.alpha;
        }
        epilogue_block(p, e, ring, v, 0, b, row_first, c0, lane, p.tri && c0 == row_first, sums);
      }
      if (!alive) break;
      if (cc_first >= cc_end) release();
      ++tile;
      if (e.stats) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sums.mabs = fmaxf(sums.mabs, __shfl_xor_sync(0xffffffffu, sums.mabs, o));
        if (lane == 0) atomicMax(p.maxabs + b, __float_as_uint(sums.mabs));
      }
      __syncwarp();
      if (ptx::elect_one()) {
        ptx::bulk_wait_all();       // this warp's part of the tile is written
        ptx::mbar_arrive(written);
      }
    }
    __syncwarp();
    if (ptx::elect_one()) {
      if (c_buf) ptx::mbar_wait(c_bar(ew), c_phase, kDrainCycles);
      ptx::bulk_wait_all();
    }
  }

  ptx::tc_fence_before();
  if constexpr (kPair) ptx::cluster_sync();
  else __syncthreads();
  if (warp == 1) {
    ptx::tc_fence_after();
    if constexpr (kPair) ptx::tmem_dealloc_pair(tmem_base, S::kTmemCols);
    else ptx::tmem_dealloc(tmem_base, S::kTmemCols);
  }
}

}  // namespace toner
