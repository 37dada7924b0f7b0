// One-sweep kernel for the decode shapes with 16 < M <= 128 queries (operand rows of at most 256
// bytes): both passes of keystream_sm100.cuh in ONE launch, so that the keys cross the HBM bus once.
//
// What bounds the shape is reading K: 2 * D bytes per key against 4 * M * D flops.  Two kernels read it
// twice (a batch's K is far larger than the L2 cache).  Here a CTA alternates between the two passes on
// small chunks of keys: record n is the rows pass of its n-th chunk, then the columns pass of
// its (n-1)-th, whose key tiles it asked for one record earlier and which therefore come from the L2
// (onesweep_chunks bounds the chunk for that).  The rows' chunk
// states of a head are exchanged through global memory: the statistics warps merge the four warpgroups'
// states of a chunk, publish them and count the chunk in a per-head counter; before a columns segment they
// wait until all chunks of its head are counted and fold them, in chunk order, into the lse values.
//
// The CTAs wait on one another, but not for CTAs that have yet to start: the TMA warp draws the chunks from a ticket
// counter and deals the records (OneSweepDealer, which has the argument), so that the call finishes on whatever SMs
// are free.  Dealt round-robin to CTAs that all had to be resident (a cooperative launch), it could not even start
// while a kernel of another stream held one SM.
//
// Measured (us per call in a graph, sustained, fp16, on one board): 16 x 32 heads, 64 x 16384, d = 128: 888 in two
// sweeps, 680 here; 8 heads, 64 x 32768: 46.6 -> 26.7; one head, 64 x 60000: 81 -> 20.5 (few heads: the combination of
// many partial states and two launches go too); 32 heads, 128 x 4096: 26.8 -> 23.3; 2 heads, 128 x 100000: 83 -> 43.
// (Dealt round-robin under a cooperative launch the same five took 674, 24.7, 20.4, 22.6 and 39: the tickets cost up to
// a tenth where a CTA has two long chunks, and nothing to speak of elsewhere.)  What bounds the large one is power: the
// board sits at its 1000 W cap with the SMs at 1.4 GHz.  On a quarter of that batch DRAM reads are 563 MB for 537 MB of
// K, MUFU is busy for 39 %, the tensor pipe for 37 %, the issue slots for 47 % of the time.
//
// Spare rows of the 128-row MMA repeat the query tile (2 copies for M <= 64, 4 for M <= 32), so that in the rows
// pass the warps of those lanes fold their own share of a key tile's columns; with one copy two of the four
// schedulers had nothing to fold.
//
// Warps: 0-15 fold (four warpgroups, one per accumulator buffer, tiles in turn), 16 loads, 17 and 18 issue
// the MMAs (tiles in turn), 19-22 keep the statistics (lane = query).
//
// Included by colreduce_sm100.cu after keystream_sm100.cuh.
#pragma once

namespace fcr {

constexpr int kOsMmaWarps = 2;  // take the tiles in turn: issuing one costs a warp about 1000 cycles with its waits, its MMAs take 256 to 512 (16 x 32 heads, 64 x 16384: 728 us with one warp, 671 with two)
constexpr int kOsStatWarp = kKsMmaWarp + kOsMmaWarps;
constexpr int kOsStatWarps = 4;
constexpr int kOsThreads = (kOsStatWarp + kOsStatWarps) * 32;
constexpr int kOsLseBuffers = 4;    // chunks whose lse values may wait for their columns segment
// Chunks whose warpgroup states may wait to be merged: one buffer per team of statistics warps, so that the uses of
// a buffer are waited for by one team, in order.
constexpr int kOsPartBuffers = 4;
// Records announced to the other warps.  The TMA warp deals one ahead; the statistics warps may lag by the part buffers.
constexpr int kOsRecords = 16;
constexpr int kOsEnd = -2;  // in the place of a head: the last record
constexpr int kOsChunk = 32;  // accumulator columns per tensor-memory load (736 threads: 80 registers)

// A missing tile shows first in its own CTA (bound 1: Q_FULL, RING_FULL, TMEM_FULL, DRAIN), then in the CTAs that wait for
// its chunk's state (HEAD: 2), last in the warps that wait behind those (3).
enum {
  ST_OS_WAIT_Q_EMPTY = 61,
  ST_OS_WAIT_RING_EMPTY = 62,
  ST_OS_WAIT_Q_FULL = 63,
  ST_OS_WAIT_RING_FULL = 64,
  ST_OS_WAIT_TMEM_EMPTY = 65,
  ST_OS_WAIT_DRAIN = 66,
  ST_OS_WAIT_TMEM_FULL = 67,
  ST_OS_WAIT_PART_EMPTY = 68,
  ST_OS_WAIT_PART_FULL = 69,
  ST_OS_WAIT_HEAD = 70,
  ST_OS_WAIT_LSE_EMPTY = 71,
  ST_OS_WAIT_LSE_FULL = 72,
  ST_OS_WAIT_RECORD_EMPTY = 73,
  ST_OS_WAIT_RECORD_FULL = 74,
};

template <int DPAD>
struct OneSweepSmem {
  static constexpr int kTileBytes = kTile * DPAD * 2;
  static constexpr int kHalves = DPAD / 64;
  static constexpr int kHalfBytes = kTile * 128;
  static constexpr int KR = DPAD == 64 ? 8 : 4;  // key tiles in flight
  static constexpr int off_q = 0;                // the query tiles of the rows and of the columns segment
  static constexpr int off_ring = off_q + 2 * kTileBytes;
  static constexpr int off_part = off_ring + KR * kTileBytes;              // float2 [kOsPartBuffers][kKsBuffers][kTile]
  static constexpr int off_lse = off_part + kOsPartBuffers * kKsBuffers * kTile * 8;    // float [kOsLseBuffers][kTile]
  static constexpr int off_bars = off_lse + kOsLseBuffers * kTile * 4;
  static constexpr int kNumBars = 4 + 2 * KR + 2 * kKsBuffers + 2 * kOsPartBuffers + 2 * kOsLseBuffers + 2 * kOsRecords;
  static constexpr int off_misc = off_bars + 8 * kNumBars;
  static constexpr int off_records = off_misc + 16;               // int4 [kOsRecords][2]: rows pass, columns pass (head, chunk, tiles)
  static constexpr int off_held = off_records + 32 * kOsRecords;  // int [kOneSweepHeld], the dealer's
  static_assert(off_records % 16 == 0, "records are read as 16 bytes");
  static constexpr int kDynamicBytes = off_held + 4 * kOneSweepHeld;
  static_assert(kDynamicBytes <= 232448, "exceeds the 227 KB shared memory of an sm_100 CTA");
};

template <int DPAD, int RED>
__global__ void __launch_bounds__(kOsThreads, 1)
onesweep_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                const PassParams p, float2* __restrict__ chunk_state, int* __restrict__ head_count,
                int* __restrict__ ticket_count, const uint32_t idesc_cols, const int copies) {
  using L = OneSweepSmem<DPAD>;
  constexpr int KR = L::KR;
  extern __shared__ __align__(1024) uint8_t smem[];
  const uint32_t base = ptx::smem_u32(smem);
  if ((base & 1023u) != 0) {
    if (threadIdx.x == 0) report_status(p, ST_SMEM_MISALIGNED, (int)base);
    return;
  }
  const uint32_t s_q = base + L::off_q;
  const uint32_t s_ring = base + L::off_ring;
  const uint32_t bar0 = base + L::off_bars;
  auto bar_q_full = [&](uint32_t kind) { return bar0 + 8u * kind; };
  auto bar_q_empty = [&](uint32_t kind) { return bar0 + 8u * (2 + kind); };
  auto bar_ring_full = [&](uint32_t s) { return bar0 + 8u * (4 + s); };
  auto bar_ring_empty = [&](uint32_t s) { return bar0 + 8u * (4 + KR + s); };
  auto bar_tm_full = [&](uint32_t b) { return bar0 + 8u * (4 + 2 * KR + b); };
  auto bar_tm_empty = [&](uint32_t b) { return bar0 + 8u * (4 + 2 * KR + kKsBuffers + b); };
  constexpr int kTail = 4 + 2 * KR + 2 * kKsBuffers;
  auto bar_part_full = [&](uint32_t i) { return bar0 + 8u * (kTail + i); };
  auto bar_part_empty = [&](uint32_t i) { return bar0 + 8u * (kTail + kOsPartBuffers + i); };
  auto bar_lse_full = [&](uint32_t i) { return bar0 + 8u * (kTail + 2 * kOsPartBuffers + i); };
  auto bar_lse_empty = [&](uint32_t i) { return bar0 + 8u * (kTail + 2 * kOsPartBuffers + kOsLseBuffers + i); };
  auto bar_rec_full = [&](uint32_t i) { return bar0 + 8u * (kTail + 2 * kOsPartBuffers + 2 * kOsLseBuffers + i); };
  auto bar_rec_empty = [&](uint32_t i) {
    return bar0 + 8u * (kTail + 2 * kOsPartBuffers + 2 * kOsLseBuffers + kOsRecords + i);
  };
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(smem + L::off_misc);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + L::off_misc + 4);
  float2* const part_s = reinterpret_cast<float2*>(smem + L::off_part);
  float* const lse_all = reinterpret_cast<float*>(smem + L::off_lse);
  int4* const records = reinterpret_cast<int4*>(smem + L::off_records);

  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);  // warp-uniform for the compiler
  const int lane = (int)(threadIdx.x & 31);
  const int live_warps = (p.M + 31) >> 5;  // statistics warps (and 32-lane groups of a query tile) that hold a query
  const int copy_rows = kTile / copies;    // rows of one copy of the query tile

  // the first ticket, asked for before the set-up so that its round trip passes meanwhile
  int first_ticket = 0;
  if (warp == kKsProducerWarp && lane == 0) first_ticket = atomicAdd(ticket_count, 1);

  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) {
      ptx::mbar_init(bar_q_full(i), 1);
      ptx::mbar_init(bar_q_empty(i), kOsMmaWarps);
    }
    for (int i = 0; i < kOsPartBuffers; ++i) {
      ptx::mbar_init(bar_part_full(i), kKsSoftmaxWarps);
      ptx::mbar_init(bar_part_empty(i), live_warps);
    }
    for (int i = 0; i < kOsLseBuffers; ++i) {
      ptx::mbar_init(bar_lse_full(i), live_warps);
      ptx::mbar_init(bar_lse_empty(i), kKsSoftmaxWarps);
    }
    for (int i = 0; i < KR; ++i) {
      ptx::mbar_init(bar_ring_full(i), 1);
      ptx::mbar_init(bar_ring_empty(i), 1);
    }
    for (int b = 0; b < kKsBuffers; ++b) {
      ptx::mbar_init(bar_tm_full(b), 1);
      ptx::mbar_init(bar_tm_empty(b), 4);
    }
    for (int i = 0; i < kOsRecords; ++i) {
      ptx::mbar_init(bar_rec_full(i), 1);
      ptx::mbar_init(bar_rec_empty(i), kKsSoftmaxWarps + kOsMmaWarps + live_warps * copies);
    }
    *abort_flag = 0;
    ptx::fence_mbar_init();
  }
  if (warp == kKsMmaWarp) {
    ptx::tmem_alloc(ptx::smem_u32(const_cast<uint32_t*>(tmem_slot)), kTmemCols);
    ptx::tmem_relinquish();
  }
  if (warp == kKsProducerWarp && lane == 0) {
    ptx::prefetch_tensormap(&tmap_q);
    ptx::prefetch_tensormap(&tmap_k);
  }
  ptx::tc_fence_before_sync();
  __syncthreads();
  ptx::tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  if (threadIdx.x == 0) ptx::grid_launch_dependents();
  if (p.clear_status && blockIdx.x == 0 && threadIdx.x < 4) p.status[threadIdx.x] = 0;

  // A record is the rows pass of one chunk (kind 0) and then the columns pass of another (kind 1), or one of them.  The
  // TMA warp decodes it once (two 64-bit divisions a chunk); the others read it where they need it and give it back.
  const int S = p.n_split;
  struct Segment { int bh, sp, t_lo, t_hi; };
  // Waits for the n-th record; false at the end, or when the wait expired (then not ok).
  auto next_record = [&](uint32_t n, bool& ok) {
    ok = WAIT_BEHIND_PEERS(bar_rec_full(n % kOsRecords), (n / kOsRecords) & 1u, ST_OS_WAIT_RECORD_FULL);
    return ok && __shfl_sync(0xffffffffu, records[2 * (n % kOsRecords)].x, 0) != kOsEnd;
  };
  auto segment = [&](uint32_t n, int kind, Segment& g) {
    const int4 v = records[2 * (n % kOsRecords) + kind];  // (shuffled: warp-uniform for the compiler)
    g.bh = __shfl_sync(0xffffffffu, v.x, 0);
    g.sp = __shfl_sync(0xffffffffu, v.y, 0);
    g.t_lo = __shfl_sync(0xffffffffu, v.z, 0);
    g.t_hi = __shfl_sync(0xffffffffu, v.w, 0);
    return g.bh >= 0;
  };
  auto record_done = [&](uint32_t n) {
    __syncwarp();
    if (lane == 0) ptx::mbar_arrive(bar_rec_empty(n % kOsRecords));
  };

  if (warp == kKsProducerWarp) {
    // ------------------------------------------------------------ TMA warp
    // A rows segment's tiles are wanted once more, a columns segment's never again: told so, the L2 gives up the
    // latter first (the large batch above took 795 to 808 us without the hint where it took 671 with it).
    const uint64_t keep = ptx::l2_policy_evict_normal(), drop = ptx::l2_policy_evict_first();
    uint32_t ring_seq = 0, q_seq[2] = {0, 0};
    bool ok = true;
    // self-test of the bounded waits: this load is left out
    const uint32_t skip_seq = blockIdx.x == 0 ? (uint32_t)p.skip_ring_load : ~0u;
    int ticket = 0;  // lane 0: the next ticket, on its way
    // one pass over a chunk: its head's query tile (a head's chunks go to different CTAs), then its key tiles
    auto load_segment = [&](const Segment& g, int kind, bool draw) {
      const int draw_at = draw ? max(g.t_lo, g.t_hi - 2) : -1;
      const int b = g.bh / p.H, h = g.bh - b * p.H;
      if (!WAIT_BEHIND_PEERS(bar_q_empty(kind), (q_seq[kind] & 1u) ^ 1u, ST_OS_WAIT_Q_EMPTY)) return false;
      if (lane == 0) {
        ptx::mbar_arrive_expect_tx(bar_q_full(kind), L::kTileBytes);
        for (int c = 0; c < copies; ++c)
#pragma unroll
          for (int hf = 0; hf < L::kHalves; ++hf)
            ptx::tma_load_4d(s_q + kind * L::kTileBytes + hf * L::kHalfBytes + c * copy_rows * 128, &tmap_q,
                             bar_q_full(kind), hf * p.slab_elems, 0, h, b);
      }
      __syncwarp();
      ++q_seq[kind];
      for (int t = g.t_lo; t < g.t_hi; ++t, ++ring_seq) {
        const uint32_t s = ring_seq % KR, ph = (ring_seq / KR) & 1u;
        if (!WAIT_BEHIND_PEERS(bar_ring_empty(s), ph ^ 1u, ST_OS_WAIT_RING_EMPTY)) return false;
        if (t == draw_at && lane == 0) ticket = atomicAdd(ticket_count, 1);
        if (ring_seq != skip_seq && ptx::elect_one()) {
          ptx::mbar_arrive_expect_tx(bar_ring_full(s), L::kTileBytes);
#pragma unroll
          for (int hf = 0; hf < L::kHalves; ++hf)
            ptx::tma_load_4d_hint(s_ring + s * L::kTileBytes + hf * L::kHalfBytes, &tmap_k, bar_ring_full(s),
                                  hf * p.slab_elems, t * kTile, h, b, kind == 0 ? keep : drop);
        }
        __syncwarp();
      }
      return true;
    };
    uint32_t n = 0;  // records so far
    OneSweepDealer dealer;
    dealer.start(S, p.n_items, reinterpret_cast<int*>(smem + L::off_held), __shfl_sync(0xffffffffu, first_ticket, 0));
    Segment r[2];  // the record dealt last
    auto announce = [&]() {
      int item[2] = {kOsEnd, -1};
      if (!dealer.finished()) dealer.deal(item[0], item[1]);
#pragma unroll
      for (int kind = 0; kind < 2; ++kind) {
        r[kind].bh = __shfl_sync(0xffffffffu, item[kind], 0);
        if (r[kind].bh >= 0)
          keystream_item(S, p.key_tiles, r[kind].bh, r[kind].bh, r[kind].sp, r[kind].t_lo, r[kind].t_hi);
      }
      const uint32_t i = n % kOsRecords;
      if (!WAIT_BEHIND_PEERS(bar_rec_empty(i), ((n / kOsRecords) & 1u) ^ 1u, ST_OS_WAIT_RECORD_EMPTY)) return false;
      if (lane == 0) {
        records[2 * i] = make_int4(r[0].bh, r[0].sp, r[0].t_lo, r[0].t_hi);
        records[2 * i + 1] = make_int4(r[1].bh, r[1].sp, r[1].t_lo, r[1].t_hi);
        ptx::mbar_arrive(bar_rec_full(i));
      }
      __syncwarp();
      ++n;
      return true;
    };
    ok = announce();
    while (ok && r[0].bh != kOsEnd) {
      const bool draw = dealer.needs_ticket(), first = n == 1;
      // Drawn with the requests of the rows pass's last tiles: not earlier, because a CTA that is a little ahead would
      // take a chunk that another SM will be free for (8 heads, 64 x 32768, two chunks per CTA: 34.7 us when drawn a
      // rows pass earlier, 26.7 here).  For the same reason a first chunk that about fits the ring draws once a tile
      // has landed: by then every CTA of the launch has had its turn.
      const bool rows = r[0].bh >= 0, small = first && rows && r[0].t_hi - r[0].t_lo <= KR + 1;
      if (rows) ok = load_segment(r[0], 0, draw && !small);
      if (ok && small && ring_seq <= KR) ok = WAIT(bar_ring_full(0), 0, ST_OS_WAIT_RING_FULL);  // (else a slot came back)
      if (!ok) break;
      if (draw && (small || !rows) && lane == 0) ticket = atomicAdd(ticket_count, 1);
      const Segment cols = r[1];
      if (draw) dealer.draw(__shfl_sync(0xffffffffu, ticket, 0));
      ok = announce();
      if (!ok) break;
      if (cols.bh >= 0) ok = load_segment(cols, 1, false);
    }
  } else if (warp < kOsStatWarp && warp >= kKsMmaWarp) {
    // ------------------------------------------------------------ MMA warps
    const uint32_t my_turn = (uint32_t)(warp - kKsMmaWarp);
    uint32_t ring_seq = 0, q_seq[2] = {0, 0};
    bool ok = true;
    for (uint32_t n = 0; ok && next_record(n, ok); ++n) {
#pragma unroll 1
      for (int kind = 0; kind < 2; ++kind) {
        Segment g;
        if (!ok || !segment(n, kind, g)) continue;
        ok = WAIT(bar_q_full(kind), (kind == 0 ? q_seq[0]++ : q_seq[1]++) & 1u, ST_OS_WAIT_Q_FULL);
        if (!ok) continue;
        ptx::tc_fence_after_sync();
        for (int t = g.t_lo; t < g.t_hi; ++t, ++ring_seq) {
          if (ring_seq % kOsMmaWarps != my_turn) continue;
          const uint32_t s = ring_seq % KR, ph = (ring_seq / KR) & 1u;
          ok = WAIT(bar_ring_full(s), ph, ST_OS_WAIT_RING_FULL);
          if (!ok) break;
          const uint32_t buf = ring_seq % kKsBuffers;
          ok = WAIT_BEHIND_PEERS(bar_tm_empty(buf), ((ring_seq / kKsBuffers) & 1u) ^ 1u, ST_OS_WAIT_TMEM_EMPTY);
          if (!ok) break;
          ptx::tc_fence_after_sync();
          if (ptx::elect_one()) {
            const uint32_t d = tmem_base + buf * kTile;
            const uint32_t k_addr = s_ring + s * L::kTileBytes;
            const uint32_t q_addr = s_q + kind * L::kTileBytes;
            // rows segment: lanes = queries (A = query tile); columns segment: lanes = keys (A = key
            // tile), and only the accumulator columns that hold a query are computed
            const uint32_t a_addr = kind == 0 ? q_addr : k_addr;
            const uint32_t b_addr = kind == 0 ? k_addr : q_addr;
            const uint32_t idesc = kind == 0 ? p.idesc : idesc_cols;
            const uint32_t a_lo = ptx::smem_desc_lo(a_addr), b_lo = ptx::smem_desc_lo(b_addr);
            auto issue_steps = [&](auto as_tf32) {
#pragma unroll
              for (int kk = 0; kk < DPAD / 16; ++kk) {
                const uint32_t koff = (uint32_t)(kk >> 2) * (L::kHalfBytes >> 4) + (uint32_t)(kk & 3) * 2u;
                ptx::umma_step<decltype(as_tf32)::value>(d, a_lo + koff, b_lo + koff, idesc, kk == 0);
              }
            };
            if (p.tf32)
              issue_steps(std::true_type{});
            else
              issue_steps(std::false_type{});
            ptx::umma_commit(bar_tm_full(buf));
            ptx::umma_commit(bar_ring_empty(s));
          }
          __syncwarp();
        }
        if (!ok) continue;
        // the query tile may be replaced once these MMAs retire
        if (ptx::elect_one()) ptx::umma_commit(bar_q_empty(kind));
        __syncwarp();
      }
      if (ok) record_done(n);
    }
    // The last commits cover every MMA issued by either warp: no asynchronous arrive is outstanding when the CTA retires.
    if (ok && q_seq[0] > 0) ok = WAIT(bar_q_empty(0), (q_seq[0] - 1) & 1u, ST_OS_WAIT_DRAIN);
    if (ok && q_seq[1] > 0) WAIT(bar_q_empty(1), (q_seq[1] - 1) & 1u, ST_OS_WAIT_DRAIN);
  } else if (warp >= kOsStatWarp) {
    // ----------------------------------------------------- statistics warps
    // A chunk's exchange is a chain of memory latencies of a few microseconds; with few queries the warps form
    // `copies` teams that take the chunks in turn, so that as many chains overlap.
    const int team_warps = kOsStatWarps / copies;
    const int team = (warp - kOsStatWarp) / team_warps, w = (warp - kOsStatWarp) % team_warps;
    const int i = w * 32 + lane;  // query
    bool ok = w < live_warps;
    // Of each record first the lse values of its columns pass, then the state of its rows pass: the fetch then starts as
    // soon as the record before it is published, a whole rows pass before the columns pass needs the values.  (It waits
    // for chunks of smaller tickets only, never for the record's own rows.)
    uint32_t n_rows = 0, n_cols = 0;  // passes so far; the teams take them in turn
    // The head of this team's last columns pass: a CTA that holds several chunks of one head folds its states once
    // (131 states took 9 us; 2 heads, 128 x 100000: 47 us without, 43 with) and copies the values of that pass.
    int lse_head = -1;
    for (uint32_t n = 0; ok && next_record(n, ok); ++n) {
      Segment g;
      if (segment(n, 1, g) && (int)(n_cols++ % copies) == team) {
        float neg_lse = lse_all[((n_cols - 1 - copies) % kOsLseBuffers) * kTile + i];
        if (g.bh != lse_head) {
          // every chunk of the head has been counted by this warp of whichever CTA folded it
          if (lane == 0) {
            const int* count = head_count + (size_t)g.bh * kOsStatWarps + w;
            if (ptx::ld_acquire(count) < S) {
              const long long t0 = clock64();
              uint32_t spins = 0;
              while (ptx::ld_acquire(count) < S) {
                if ((++spins & 7u) == 0) {
                  if (*abort_flag) {
                    ok = false;
                    break;
                  }
                  if (clock64() - t0 > 2 * p.wait_limit) {
                    *abort_flag = 1;
                    report_status(p, ST_OS_WAIT_HEAD, g.bh);
                    ok = false;
                    break;
                  }
                }
              }
            }
          }
          __syncwarp();  // lane 0's acquire covers the loads of all lanes (a vote orders no memory)
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          float mx = -INFINITY, l = 0.f;
          if (i < p.M) {
            const float2* st = chunk_state + (size_t)g.bh * p.m_pad + i;
            const size_t step = (size_t)p.BH * p.m_pad;
            constexpr int kBatch = 16;  // loads in flight
            for (int s0 = 0; s0 < S; s0 += kBatch) {
              float2 v[kBatch];
              float top = mx;
#pragma unroll
              for (int u = 0; u < kBatch; ++u)
                v[u] = s0 + u < S ? __ldcg(st + (size_t)(s0 + u) * step) : make_float2(-INFINITY, 0.f);
#pragma unroll
              for (int u = 0; u < kBatch; ++u) top = fmaxf(top, v[u].x);
              if (mx != -INFINITY) l *= exp2f(mx - top);
              mx = top;
#pragma unroll
              for (int u = 0; u < kBatch; ++u)  // a chunk this query does not see left (-inf, 0)
                if (v[u].x != -INFINITY || v[u].y != 0.f) l = fmaf(v[u].y, exp2f(v[u].x - mx), l);
            }
          }
          lse_head = g.bh;
          neg_lse = i < p.M ? -(mx + log2f(l)) : 0.f;
        }
        const uint32_t lb = (n_cols - 1) % kOsLseBuffers, lph = ((n_cols - 1) / kOsLseBuffers) & 1u;
        ok = WAIT_BEHIND_PEERS(bar_lse_empty(lb), lph ^ 1u, ST_OS_WAIT_LSE_EMPTY);
        if (!ok) break;
        lse_all[lb * kTile + i] = neg_lse;
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(bar_lse_full(lb));
      }
      if (segment(n, 0, g) && (int)(n_rows++ % copies) == team) {
        const uint32_t pb = (n_rows - 1) % kOsPartBuffers, pph = ((n_rows - 1) / kOsPartBuffers) & 1u;
        ok = WAIT_BEHIND_PEERS(bar_part_full(pb), pph, ST_OS_WAIT_PART_FULL);
        if (!ok) break;
        // the four warpgroups' states of this chunk, in the order of their tiles
        const float2* cell = part_s + pb * (kKsBuffers * kTile) + i;
        float mx = -INFINITY, l = 0.f;
        for (int c = 0; c < copies; ++c)
#pragma unroll
          for (int j = 0; j < kKsBuffers; ++j) mx = fmaxf(mx, cell[j * kTile + c * copy_rows].x);
        for (int c = 0; c < copies; ++c)
#pragma unroll
          for (int j = 0; j < kKsBuffers; ++j) {
            const float2 st = cell[j * kTile + c * copy_rows];
            if (st.x != -INFINITY || st.y != 0.f) l = fmaf(st.y, exp2f(st.x - mx), l);
          }
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(bar_part_empty(pb));
        if (i < p.M) __stcg(chunk_state + ((size_t)g.sp * p.BH + g.bh) * p.m_pad + i, make_float2(mx, l));
        __syncwarp();  // lane 0's release covers the stores of all lanes
        if (lane == 0) ptx::red_release_add(head_count + (size_t)g.bh * kOsStatWarps + w, 1);
        __syncwarp();
      }
      record_done(n);
    }
  } else {
    // -------------------------------------------------------- softmax warps
    // Warpgroup wg folds the tiles that land in accumulator buffer wg: the CTA's tile number mod 4.
    const int wg = warp >> 2;
    const int tid_wg = (warp & 3) * 32 + lane;
    const uint32_t taddr = tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)wg * kTile;
    // rows pass: this warp's lanes hold queries first_q.. (of copy `copy` of the query tile) and fold the
    // columns [col0, col0 + copy_rows) of a key tile
    const int copy = (warp & 3) * 32 / copy_rows, first_q = (warp & 3) * 32 - copy * copy_rows;
    const int col0 = copy * copy_rows;
    const bool live = first_q < p.M;
    uint32_t seq = 0, n_rows = 0, n_cols = 0;  // tiles and segments so far
    bool ok = true;
    for (uint32_t n = 0; ok && next_record(n, ok); ++n) {
#pragma unroll 1  // (unrolled, the sum reduction spills two of its 80 registers)
      for (int kind = 0; kind < 2; ++kind) {
        Segment g;
        if (!ok || !segment(n, kind, g)) continue;
        const int j0 = (int)((uint32_t)(wg - (int)seq) & (kKsBuffers - 1));  // my first tile within the chunk
        const uint32_t seq0 = seq;
        seq += (uint32_t)(g.t_hi - g.t_lo);
        if (kind == 0) {
          const int mine = first_q + lane;  // query row
          float m_run = -INFINITY, l_run = 0.f;
          // keys j < valid_hi are attended by this query; tiles from mask_from on meet a mask edge
          const int valid_hi = p.causal ? (int)hd_min((long long)p.N, (long long)mine + p.off + 1) : p.N;
          int mask_from = p.N >> 7;
          if (p.causal) mask_from = (int)hd_min((long long)mask_from, ((long long)p.off + 1) >> 7);
          for (int t = g.t_lo + j0; t < g.t_hi; t += kKsBuffers) {
            const uint32_t use = (seq0 + (uint32_t)(t - g.t_lo)) / kKsBuffers;
            ok = WAIT(bar_tm_full(wg), use & 1u, ST_OS_WAIT_TMEM_FULL);
            if (!ok) break;
            if (!live) {
              if (lane == 0) ptx::mbar_arrive(bar_tm_empty(wg));
              __syncwarp();
              continue;
            }
            ptx::tc_fence_after_sync();
            const bool need_mask = t >= mask_from;
            const int lim_hi = valid_hi - t * kTile - col0;
            const int n_fold = copy_rows / kOsChunk;
            uint32_t ra[kOsChunk];
            for (int c = 0; c < n_fold; ++c) {
              ptx::tmem_ld<kOsChunk>(taddr + col0 + c * kOsChunk, ra);
              ptx::tmem_ld_wait<kOsChunk>(ra);
              if (c + 1 == n_fold) {
                ptx::tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive(bar_tm_empty(wg));
              }
              if (need_mask)
                rows_chunk<true, kOsChunk>(ra, p.scale2, lim_hi - kOsChunk * c, m_run, l_run);
              else
                rows_chunk<false, kOsChunk>(ra, p.scale2, kOsChunk, m_run, l_run);
            }
          }
          if (!ok) break;
          const uint32_t pb = n_rows % kOsPartBuffers, pph = (n_rows / kOsPartBuffers) & 1u;
          ++n_rows;
          ok = WAIT_BEHIND_PEERS(bar_part_empty(pb), pph ^ 1u, ST_OS_WAIT_PART_EMPTY);
          if (!ok) break;
          // a warpgroup without a tile in this chunk leaves (-inf, 0), which the merge skips
          if (live) part_s[(pb * kKsBuffers + j0) * kTile + tid_wg] = make_float2(m_run, l_run);
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive(bar_part_full(pb));
        } else {
          const uint32_t lb = n_cols % kOsLseBuffers, lph = (n_cols / kOsLseBuffers) & 1u;
          ++n_cols;
          ok = WAIT_BEHIND_PEERS(bar_lse_full(lb), lph, ST_OS_WAIT_LSE_FULL);
          if (!ok) break;
          const float* lse_s = lse_all + lb * kTile;
          const int n_fold = p.fold_cols / kChunkCols;  // only the chunks that hold a query
          for (int t = g.t_lo + j0; t < g.t_hi; t += kKsBuffers) {
            const uint32_t use = (seq0 + (uint32_t)(t - g.t_lo)) / kKsBuffers;
            ok = WAIT(bar_tm_full(wg), use & 1u, ST_OS_WAIT_TMEM_FULL);
            if (!ok) break;
            ptx::tc_fence_after_sync();
            const int mine = t * kTile + tid_wg;  // key column
            float acc[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) acc[u] = (RED == RED_MAX) ? -INFINITY : 0.f;
            // queries max(mine - off, 0) <= i < M attend this key
            const int valid_lo = p.causal ? max(mine - p.off, 0) : 0;
            const bool need_mask = (p.M < p.fold_cols) || (p.causal && t * kTile + kTile - 1 - p.off > 0);
            uint32_t ra[kChunkCols];
            for (int c = 0; c < n_fold; ++c) {
              ptx::tmem_ld<kChunkCols>(taddr + c * kChunkCols, ra);
              ptx::tmem_ld_wait<kChunkCols>(ra);
              if (c + 1 == n_fold) {
                ptx::tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive(bar_tm_empty(wg));
              }
              if (need_mask)
                cols_chunk<RED, true, kChunkCols>(ra, lse_s + kChunkCols * c, p.scale2, valid_lo - kChunkCols * c,
                                                  p.M - kChunkCols * c, acc);
              else
                cols_chunk<RED, false, kChunkCols>(ra, lse_s + kChunkCols * c, p.scale2, 0, kChunkCols, acc);
            }
            if (mine < p.N) {
              float v;
              if (RED == RED_SUM)
                v = (acc[0] + acc[1]) + (acc[2] + acc[3]);
              else
                v = ptx::ex2(fmaxf(fmaxf(acc[0], acc[1]), fmaxf(acc[2], acc[3])));
              if (p.mean_mode) v = v / mean_divisor(p, mine);
              store_out(p.out, p.out_dtype, (size_t)g.bh * p.N + mine, v);
            }
          }
          if (!ok) break;
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive(bar_lse_empty(lb));  // done with these lse values
        }
      }
      if (ok) record_done(n);
    }
  }

  // ------------------------------------------------------------- teardown
  __syncwarp();
  ptx::tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag) {
    // A wait expired somewhere: give loads that may still be in flight time to
    // land in this CTA's shared memory before it is released.
    for (int k = 0; k < 2000; ++k) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == kKsMmaWarp) {
    ptx::tc_fence_after_sync();
    ptx::tmem_dealloc(tmem_base, kTmemCols);
  }
}

}  // namespace fcr
