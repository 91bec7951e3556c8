// vfb_kernels.cu -- sm_100a kernels of one level step of the cached search.
//
// Every kernel reads its work from device memory, so the same launch
// sequence serves every level and any number of instances.  The graph solver
// builds level k with
//
//   k_p1          every candidate: operator words -> 126-bit key -> insert
//                 into the instance's hash set with atomicMin on the
//                 candidate's canonical index; the smallest candidate index
//                 whose CS satisfies the sample is recorded
//                 (applyOperator LTL_BS.cu:183-238, makeRlxUnqChkCSs 30-110,
//                  processUniqueCS 251-269)
//   k_table_scan_check
//                 a slot whose final payload carries level k holds a key first
//                 seen at this level; its payload's index is the key's owner
//                 (the minimum candidate index): set the owner's bit.  Also
//                 settles whether the recorded solution candidate owns its key
//                 and checks the level's buffers; of a few instances' small
//                 levels it compacts the bitmap too
//   k_compact     ordered compaction of the owner bitmap into the ascending
//                 owner list
//   k_emit        the owners' rows appended to the level cache in canonical
//                 order, solution test (insertInCache LTL_BS.cu:299-329); rows
//                 skipped when the solution is settled
//   k_advance     level bookkeeping, formula reconstruction (LTL_BS.cu:561-705),
//                 then the next level's candidate-block bases, P1 tiling and
//                 buffer checks (LTL_BS.cu:1226-1488)
//
// The persistent and cluster solvers run the same phases (plan, P1, table
// scan, chunk count/scan/emit, row emission, finish) inside one kernel, between
// barriers.
//
// The reference's thrust::remove/copy_n compaction (storeUniqueLTLs
// LTL_BS.cu:489-530) is replaced by the bitmap compaction; its racy
// atomicCAS winners (LTL_BS.cu:319, hash_set.cuh:232) by min-index ownership.
#include <cooperative_groups.h>

#include "vfb_ops.cuh"

namespace vfb {

// Programmatic dependent launch inside the level step: wait until the
// preceding kernel has completed and its writes are visible, then let the
// next kernel be scheduled while this one runs (its CTAs then wait here
// themselves).  Both are no-ops for a launch without the attribute.
__device__ __forceinline__ void step_entry() {
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
}

// Few instances at a time: the table scan takes only the CTAs that the levels'
// lists need (a small level's list is one CTA's: no ticket, no waiting for
// idle ones).
__device__ __forceinline__ bool scan_compacts(const BatchDev& B) { return B.ninst <= 4; }
// Whether the owner bitmap of an instance's level is compacted by the last CTA
// of the table scan (256 threads, two words each) instead of by k_compact: a
// kernel's start, ticket and look-back (4-5 us) cost more than the level's one
// chunk.  One CTA would take the instances of a batch in turn: few only.
__device__ __forceinline__ bool small_compact(const BatchDev& B, uint64_t plan_words) {
  return scan_compacts(B) && plan_words <= kCompactWords;
}

// ===================================================================== plan
// Plan level k = I.level of a RUNNING instance: candidate-block bases, P1
// tiling, buffer checks.  Records the plan (planned = k, plan_*) or asks the
// host for memory (NEED_MEM, planned = 0).
__device__ void plan_one(InstDev& I, bool few) {
  // Everything the plan reads is loaded first: the plan runs on one thread,
  // and a load issued after a store to the record waits for that store.
  const int k = I.level, weighted = I.weighted, on_the_fly = I.on_the_fly;
  const int c1 = atom_level(I), Ln = not_level(I, k);
  const int wA = op_cost(I, OP_AND), wO = op_cost(I, OP_OR), wX = op_cost(I, OP_X), wF = op_cost(I, OP_F),
            wG = op_cost(I, OP_G), wU = op_cost(I, OP_U);
  uint64_t n[kMaxSize + 1];
  for (int i = 0; i <= k; ++i) n[i] = I.lcount[i];
  const uint64_t lstart_prev = I.lstart[k - 1];
  const uint64_t keys = I.keys, table_cap = I.table_mask + 1, bitmap_words = I.bitmap_words,
                 row_cap = I.row_cap, tent_cap = I.tent_cap, promote_above = I.promote_above;
  static_assert(kTS == 1 << 7, "");
  const bool by_words = !exact_keys(I) && I.TP >= 8;   // (keys that take every word)
  const uint64_t split_tiles = kP1SplitTiles * (I.TP > 64 ? 8 : 1);
  const int attempt = I.attempt, attempt_level = I.attempt_level, rows_deferred = I.rows_deferred;
  const int no_mask = (attempt_level == k) ? I.no_mask : 0;
  // the first operand rows whose ~ X F G candidates satisfy the sample
  // (recorded when those rows were written)
  const int ulev[4] = {Ln, k - wX, k - wF, k - wG};
  uint32_t uh[4];
#pragma unroll
  for (int o = 0; o < 4; ++o) uh[o] = ulev[o] >= c1 ? I.uhit[ulev[o]][o] : 0u;
  const uint64_t lstart_k = lstart_prev + n[k - 1];
  I.lstart[k] = lstart_k;
  // candidate blocks in canonical order: ~ & | X F G U; a unary operator of
  // cost c reads level k - c, & | over splits (i, k - c - i) with i <= k - c - i,
  // U over every split (LTL_BS.cu:1226-1488; unit costs: the size order)
  uint64_t g = 0;
  uint64_t bA[kMaxSize + 1], bO[kMaxSize + 1], bU[kMaxSize + 1];   // block bases by left level
  I.base_not = g;
  if (Ln >= 0) g += n[Ln];
  for (int pass = 0; pass < 2; ++pass) {
    const int w = pass ? wO : wA;
    for (int i = c1; 2 * i <= k - w; ++i) {
      const int j = k - w - i;
      (pass ? bO : bA)[i] = g;
      (pass ? I.base_or : I.base_and)[i] = g;
      g += n[i] * n[j];
    }
  }
  uint64_t bx[3];
  {
    const int ws[3] = {wX, wF, wG};
#pragma unroll
    for (int o = 0; o < 3; ++o) {
      const int L = k - ws[o];
      bx[o] = g;
      if (L >= c1) g += n[L];
    }
    I.base_x = bx[0];
    I.base_f = bx[1];
    I.base_g = bx[2];
  }
  for (int i = c1; k - wU - i >= c1; ++i) {
    bU[i] = g;
    I.base_u[i] = g;
    g += n[i] * n[k - wU - i];
  }
  I.cands = g;
  // operand groups: the unary operators by operand level (bits ~ X F G), the
  // binary ones by level pair la <= lb (bits &, |, la U lb, lb U la); with
  // unit costs one unary group and one group per split, as the reference's
  // launches fuse them.  The tiles of every staged height 2^0..2^4 (kTQ) are
  // summed on the way.
  int ng = 0;
  constexpr int kHeights = 5;
  static_assert(1 << (kHeights - 1) == kTQ, "");
  uint64_t tl[kHeights] = {0, 0, 0, 0, 0}, tsplit = 0;   // (tsplit: kTS/4 rows a tile, one staged)
  auto add_tiles = [&](int kind, int la, int lb) {
    if (kind == 0) {
      const uint64_t st = (n[la] + kTS - 1) / kTS;
      tsplit += (n[la] + kTS / 4 - 1) / (kTS / 4);
#pragma unroll
      for (int u = 0; u < kHeights; ++u) tl[u] += (st + (1ULL << u) - 1) >> u;
    } else {
      const bool qleft = (la == lb) || (n[la] <= n[lb]);
      const uint64_t nS = qleft ? n[lb] : n[la], nQ = qleft ? n[la] : n[lb];
      const uint64_t st = (nS + kTS - 1) / kTS;
      tsplit += (nS + kTS / 4 - 1) / (kTS / 4) * nQ;
#pragma unroll
      for (int u = 0; u < kHeights; ++u) tl[u] += st * ((nQ + (1ULL << u) - 1) >> u);
    }
  };
  // unit costs: one group per size split, then one unary group over level
  // k-1.  The unary group comes last so that a solution among the & | blocks,
  // which precede X F G in the candidate order, is known before its tiles
  // start: they then compute ~ alone.
  const int msplit = (k - 1) / 2;
  auto u_kind = [&](int q) { return q < msplit ? 1 : 0; };
  auto u_la = [&](int q) { return q < msplit ? q + 1 : k - 1; };
  auto u_lb = [&](int q) { return q < msplit ? k - 2 - q : 0; };
  auto u_mask = [&](int q) { return q < msplit ? (2 * (q + 1) == k - 1 ? 7 : 15) : 0xF; };
  if (!weighted) {
    for (ng = 0; ng <= msplit; ++ng) {
      I.grp_kind[ng] = (uint8_t)u_kind(ng);
      I.grp_la[ng] = (uint8_t)u_la(ng);
      I.grp_lb[ng] = (uint8_t)u_lb(ng);
      I.grp_mask[ng] = (uint8_t)u_mask(ng);
      add_tiles(u_kind(ng), u_la(ng), u_lb(ng));
    }
  } else {
    // weighted: a level (pair) may serve several operators, so the groups
    // are collected first, then their tiles summed
    auto unary = [&](int L, int bit) {
      if (L < c1) return;
      for (int q = 0; q < ng; ++q)
        if (I.grp_kind[q] == 0 && I.grp_la[q] == L) { I.grp_mask[q] |= (uint8_t)(1 << bit); return; }
      if (ng >= kGroups) return;
      I.grp_kind[ng] = 0; I.grp_la[ng] = (uint8_t)L; I.grp_lb[ng] = 0; I.grp_mask[ng] = (uint8_t)(1 << bit);
      ++ng;
    };
    auto binary = [&](int la, int lb, int bits) {
      for (int q = 0; q < ng; ++q)
        if (I.grp_kind[q] == 1 && I.grp_la[q] == la && I.grp_lb[q] == lb) { I.grp_mask[q] |= (uint8_t)bits; return; }
      if (ng >= kGroups) return;
      I.grp_kind[ng] = 1; I.grp_la[ng] = (uint8_t)la; I.grp_lb[ng] = (uint8_t)lb; I.grp_mask[ng] = (uint8_t)bits;
      ++ng;
    };
    unary(Ln, 0);
    unary(k - wX, 1);
    unary(k - wF, 2);
    unary(k - wG, 3);
    const int s3 = k - wA, s4 = k - wO, s8 = k - wU;
    const int sums[3] = {s3, s4, s8};
    for (int q = 0; q < 3; ++q) {
      const int sm = sums[q];
      if (q == 1 && sm == s3) continue;
      if (q == 2 && (sm == s3 || sm == s4)) continue;
      for (int i = c1; 2 * i <= sm; ++i) {
        const int j = sm - i;
        int bits = 0;
        if (sm == s3) bits |= 1;
        if (sm == s4) bits |= 2;
        if (sm == s8) bits |= (i == j) ? 4 : (4 | 8);
        binary(i, j, bits);
      }
    }
    for (int q = 0; q < ng; ++q) add_tiles(I.grp_kind[q], I.grp_la[q], I.grp_lb[q]);
  }
  I.ngroups = ng;
  // operator bases of every group (what a P1 tile needs to tell whether an
  // operator's candidates can still come before the best solution found)
  for (int q = 0; q < ng; ++q) {
    const int kind = weighted ? I.grp_kind[q] : u_kind(q);
    const int mask = weighted ? I.grp_mask[q] : u_mask(q);
    const int la = weighted ? I.grp_la[q] : u_la(q);
    const int lb = weighted ? I.grp_lb[q] : u_lb(q);
    uint64_t b4[4];
    if (kind == 0) {
      b4[0] = 0;   // ~ is the first block
      b4[1] = bx[0];
      b4[2] = bx[1];
      b4[3] = bx[2];
    } else {
      b4[0] = (mask & 1) ? bA[la] : 0;
      b4[1] = (mask & 2) ? bO[la] : 0;
      b4[2] = (mask & 4) ? bU[la] : 0;
      b4[3] = (mask & 8) ? bU[lb] : 0;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) I.grp_base[q][u] = b4[u];
  }
  // P1 tiling: kTS stream rows x tq staged rows per tile, or tq blocks of kTS
  // rows of a unary group (about the same work).  The height
  // is the largest power of two within the band's bound whose tile count
  // reaches the band's target (small levels get shorter tiles so that they
  // still spread over every SM and end in a short last wave), else 1.  The
  // level's band of the tune table also sets the CTAs to launch.
  const int band = tune_band(g);
  const int rows_max = p1_rows_max(I.TP);
  const int rows_want = I.tune_rows[band] ? I.tune_rows[band] : kTQDefault;
  const int rows_cap = rows_want < rows_max ? rows_want : rows_max;
  const uint64_t target = I.tune_tiles[band] ? 1ULL << I.tune_tiles[band] : (uint64_t)kP1TileTarget;
  I.p1_blocks = I.tune_blocks[band];
  int lg = 0;
  uint64_t t = tl[0];
#pragma unroll
  for (int u = 1; u < kHeights; ++u)
    if ((1 << u) <= rows_cap && tl[u] >= target) { lg = u; t = tl[u]; }
  I.tq = 1 << lg;
  // four lanes to a stream row where the level then still runs in one wave
  // (see kP1SplitTiles; in a batch the other instances fill the SMs)
  const int split = few && by_words && !on_the_fly && lg == 0 && tsplit <= split_tiles ? 2 : 0;
  const uint64_t height = kTS >> split;
  if (split) t = tsplit;
  I.p1_split = split;
  // group boundaries in tiles (ph_p1 reads the first ngroups of them)
  {
    uint64_t acc = 0;
    I.grp_prefix[0] = 0;
    for (int q = 0; q < ng; ++q) {
      const int kind = weighted ? I.grp_kind[q] : u_kind(q);
      const int la = weighted ? I.grp_la[q] : u_la(q);
      const int lb = weighted ? I.grp_lb[q] : u_lb(q);
      if (kind == 0) {
        acc += (((n[la] + height - 1) >> (7 - split)) + (1ULL << lg) - 1) >> lg;
      } else {
        const bool qleft = (la == lb) || (n[la] <= n[lb]);
        const uint64_t nS = qleft ? n[lb] : n[la], nQ = qleft ? n[la] : n[lb];
        const uint64_t qt = (nQ + (1ULL << lg) - 1) >> lg, st = (nS + height - 1) >> (7 - split);
        I.grp_qtiles[q] = (uint32_t)qt;
        acc += st * qt;
      }
      I.grp_prefix[q + 1] = acc;
    }
  }
  const uint64_t words = on_the_fly ? 0 : (g + 31) / 32;
  // new keys of this level: at most all candidates; expect ~8x growth
  const uint64_t grow = 8 * n[k - 1] + 4096;
  const uint64_t est = g < grow ? g : grow;
  int need = 0;
  if (g >= (1ULL << kPayShift)) need |= NEED_LIMIT;
  if (!on_the_fly) {   // an on-the-fly level stores nothing
    if (g > promote_above) need |= NEED_PROMOTE;
    if (words > bitmap_words) { need |= NEED_BITMAP; I.need_amount[0] = words; }
    // (twice the projected keys, rounded up to a power of two: at most half
    // full if the projection holds; 4x measured 6% slower on large
    // instances, from filling and rehashing twice the bytes)
    if (2 * (keys + est) > table_cap) { need |= NEED_TABLE; I.need_amount[1] = 2 * (keys + est); }
    // (a projection the host cannot hold is deferred: the table scan asks for
    // the rows the level's owners need, none when it settles the solution)
    if (!rows_deferred && lstart_k + est > row_cap) {
      need |= NEED_ROWS | NEED_ROWS_EST;
      I.need_amount[3] = lstart_k + est;
    }
    if (est > tent_cap) { need |= NEED_LIST; I.need_amount[2] = est; }
  }
  if (need) {
    I.status = ST_NEED_MEM;
    I.need = need;
    I.planned = 0;
  } else {
    I.plan_tiles = t;
    I.plan_words = words;
    // scan chunks of kScanSlots, larger on larger tables (8 kScanSlots while
    // 2048 chunks remain, 32 while 8192 do): small levels spread over the SMs,
    // large ones make fewer per-chunk reductions and atomics; the instances of
    // a batch fill the SMs together and start at 8 kScanSlots
    uint64_t ss = (few ? 1 : 8) * (uint64_t)kScanSlots;
    while (ss < 8 * (uint64_t)kScanSlots && table_cap / (2 * ss) >= 2048) ss *= 2;
    while (ss < 32 * (uint64_t)kScanSlots && table_cap / (2 * ss) >= 8192) ss *= 2;
    I.scan_slots = (uint32_t)ss;
    I.plan_tchunks = on_the_fly ? 0 : (table_cap + ss - 1) / ss;
    I.planned = k;
    I.p1_done = 0;
    I.p1_step = t;
    I.p1_tail = 1;
    I.n_new = I.n_wins = I.probe_fail = I.n_newlist = 0;
    // A unary candidate recorded as satisfying the sample bounds the level's
    // first solution from the start, as if a P1 tile had found it: operators
    // past it are skipped everywhere (not in a full re-run)
    uint64_t first = ~0ULL;
    if (!no_mask) {
      const uint64_t ub[4] = {0, bx[0], bx[1], bx[2]};
#pragma unroll
      for (int o = 0; o < 4; ++o) {
        const uint64_t row = 0xFFFFFFFFull - uh[o];
        if (uh[o] && row < n[ulev[o]] && ub[o] + row < first) first = ub[o] + row;
      }
    }
    I.best_cand = first;
    // a level with a solution from the start and millions of candidates before
    // it: P1 skips listing its new slots (one atomic per warp and candidate
    // group) and the table scan reads the whole table instead
    I.no_list = (first != ~0ULL && first >= (1ULL << 22)) ? 1 : 0;
    I.best_sol = ~0ULL;
    I.n_below = 0;
    I.counted_below = 0;
#pragma unroll
    for (int o = 0; o < 4; ++o) I.uhit[k][o] = 0u;   // (this level's rows are written after it)
    I.sol_known = 0;
    I.p1_masked = 0;
    if (attempt_level != k) I.no_mask = 0;   // a new level may skip again
    I.attempt = (attempt_level == k) ? attempt + 1 : 1;
    I.attempt_level = k;
  }
}

__device__ void ph_plan(const BatchDev& B, unsigned bid, unsigned nb) {
  for (int b = bid * blockDim.x + threadIdx.x; b < B.ninst; b += nb * blockDim.x) {
    InstDev& I = B.inst[b];
    unsigned long long tiles = 0, chunks = 0, tchunks = 0;
    if (I.status == ST_RUNNING) {
      plan_one(I, scan_compacts(B));
      if (I.status == ST_RUNNING) {
        tiles = I.plan_tiles;
        chunks = (I.plan_words + kChunkWords - 1) / kChunkWords;
        tchunks = I.plan_tchunks;
      }
    }
    B.p1_prefix[b + 1] = tiles;
    B.chunk_prefix[b + 1] = chunks;
    B.tscan_prefix[b + 1] = tchunks;
  }
}

// One thread: cross-instance prefixes of P1 tiles and bitmap chunks; resets
// the work tickets of the step.
__device__ void ph_plan_prefix(const BatchDev& B) {
  B.p1_prefix[0] = 0;
  B.chunk_prefix[0] = 0;
  B.tscan_prefix[0] = 0;
  for (int b = 0; b < B.ninst; ++b) {
    B.p1_prefix[b + 1] += B.p1_prefix[b];
    B.chunk_prefix[b + 1] += B.chunk_prefix[b];
    B.tscan_prefix[b + 1] += B.tscan_prefix[b];
  }
  for (int i = 0; i < kTickets; ++i) B.tickets[i] = 0;
}

// ======================================================================= P1
// The instance's part of a tile's shared parameters (thread per trace, threads
// t0 .. kTS-1), kept while a CTA's consecutive tiles are of one instance.
__device__ void p1_instance(const InstDev& I, TileSh& P, int t0) {
  const int T = I.T, TP = I.TP;
  for (int t = threadIdx.x - t0; t < TP; t += kTS - t0) {
    const int L = t < T ? I.len[t] : 0;
    P.len[t] = (uint8_t)L;
    P.tr[t] = TraceSh{len_mask(L), t < T && is_pos(I, t) ? 1u : 0u, 0u};
    P.off[t] = t < T ? I.off[t] : 0;
    P.wid[t] = t < T ? I.width[t] : 0;
  }
  if (exact_keys(I) && threadIdx.x < t0 + 32) {
    // masks over the key bits: a lane takes some traces, then XOR shuffles
    KeyAcc full{0, 0}, last{0, 0}, first{0, 0}, want{0, 0};
    for (int t = threadIdx.x - t0; t < T; t += 32) {
      const int L = I.len[t], off = I.off[t];
      key_word<KEY_CONCAT>(full, len_mask(L), t, 0, off, L, 1, L);
      key_word<KEY_CONCAT>(last, 1ULL << (L - 1), t, 0, off, L, 1, L);
      key_word<KEY_CONCAT>(first, 1ULL, t, 0, off, L, 1, L);
      key_word<KEY_CONCAT>(want, is_pos(I, t) ? 1ULL : 0ULL, t, 0, off, L, 1, L);
    }
    uint64_t v[8] = {full.a0, full.a1, last.a0, last.a1, first.a0, first.a1, want.a0, want.a1};
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] ^= __shfl_xor_sync(0xffffffffu, v[j], o);
    if (threadIdx.x == t0) {
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        P.full[j] = v[j];
        P.last[j] = v[2 + j];
        P.first[j] = v[4 + j];
        P.want[j] = v[6 + j];
      }
    }
  }
}

// The tile's staged rows into shared memory: their words (QWord) unless the
// key bits alone settle the candidates, and their key bits (QKey) where keys
// are bit fields.
__device__ __forceinline__ void p1_stage(const TileSh& P, QWord* sQ, QKey* sK) {
  const uint64_t* src = P.qrows;
  const int T = P.T, TP = P.TP;
  if (P.otf || !P.exact) {
    // (nq rows of TP words: one block, the padding words zero)
    const int dc = blockDim.x % TP;
    int c = threadIdx.x % TP;
    for (int x = threadIdx.x; x < P.nq * TP; x += blockDim.x) {
      const uint64_t w = ld_row1(src + x);
      sQ[x] = QWord{w, w >> 30, __brevll(w), P.tr[c].lab, 0u};
      c += dc;
      if (c >= TP) c -= TP;
    }
  }
  if (P.mode != KEY_HASH && !P.otf && !P.split) {
    const int lane = threadIdx.x & 31;
    for (int r = threadIdx.x >> 5; r < P.nq; r += blockDim.x >> 5) {
      KeyAcc k;
      key_init(k);
      for (int t = lane; t < T; t += 32) {
        const uint64_t w = ld_row1(src + (size_t)r * P.TP + t);
        if (P.mode == KEY_SAMPLED) key_word<KEY_SAMPLED>(k, w, t, 0, P.off[t], P.wid[t], P.stride, P.len[t]);
        else key_word<KEY_CONCAT>(k, w, t, 0, P.off[t], P.wid[t], P.stride, P.len[t]);
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        k.a0 ^= __shfl_xor_sync(0xffffffffu, k.a0, o);
        k.a1 ^= __shfl_xor_sync(0xffffffffu, k.a1, o);
      }
      if (lane == 0) sK[r] = QKey{k.a0, k.a1, __brevll(k.a1), __brevll(k.a0)};
    }
  }
}

// A tile's parameters (warp 0; local: the tile's number within its instance's
// level).  A chain of dependent loads is what this costs, so everything that
// does not depend on the tile's group is read at once, one entry per lane for
// the levels and the groups, then the group's bases.
__device__ __forceinline__ void p1_setup(InstDev* Ip, int b, uint64_t local, TileSh& P) {
  const int lane = threadIdx.x & 31;
  const int e1 = 2 * lane + 1, e2 = 2 * lane + 2;
  const uint64_t done = __ldcg(&Ip->p1_done);
  const int ngr = __ldcg(&Ip->ngroups);
  uint64_t gp1 = e1 < kGroups ? __ldcg(&Ip->grp_prefix[e1]) : ~0ULL;
  uint64_t gp2 = e2 < kGroups ? __ldcg(&Ip->grp_prefix[e2]) : ~0ULL;
  const uint64_t cnt_l = __ldcg(&Ip->lcount[lane]), start_l = __ldcg(&Ip->lstart[lane]);
  unsigned gr[2];   // groups lane, lane + 32: kind | mask << 8 | la << 16 | lb << 24
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int q = lane + 32 * u;
    gr[u] = (unsigned)__ldcg(&Ip->grp_kind[q]) | ((unsigned)__ldcg(&Ip->grp_mask[q]) << 8) |
            ((unsigned)__ldcg(&Ip->grp_la[q]) << 16) | ((unsigned)__ldcg(&Ip->grp_lb[q]) << 24);
  }
  const int k = __ldcg(&Ip->level), T = __ldcg(&Ip->T), TP = __ldcg(&Ip->TP);
  const int stride = __ldcg(&Ip->stride1), mode = __ldcg(&Ip->key_mode), tq = __ldcg(&Ip->tq);
  const int exact = __ldcg(&Ip->exact), otf = __ldcg(&Ip->on_the_fly), nolist = __ldcg(&Ip->no_list);
  const int split = __ldcg(&Ip->p1_split), height = kTS >> split;
  Slot* const table = (Slot*)__ldcg((const unsigned long long*)&Ip->table);
  const uint64_t* const rows = (const uint64_t*)__ldcg((const unsigned long long*)&Ip->rows);
  const unsigned long long tmask = __ldcg(&Ip->table_mask), keys = __ldcg(&Ip->keys);
  const unsigned long long fails = __ldcg(&Ip->probe_fail), fresh = __ldcg(&Ip->n_new);
  const unsigned long long best = __ldcg(&Ip->best_cand);
  const int may_skip = !__ldcg(&Ip->no_mask);
  // lane l holds group boundaries 2l+1 and 2l+2; the group is the number of
  // boundaries at or below the tile (boundaries past the level's groups are
  // stale: read as never reached)
  local += done;
  if (e1 >= ngr) gp1 = ~0ULL;
  if (e2 >= ngr) gp2 = ~0ULL;
  const int grp = __popc(__ballot_sync(0xffffffffu, gp1 <= local)) + __popc(__ballot_sync(0xffffffffu, gp2 <= local));
  const int src = grp >= 1 ? (grp - 1) >> 1 : 0;
  const uint64_t s1 = __shfl_sync(0xffffffffu, gp1, src), s2 = __shfl_sync(0xffffffffu, gp2, src);
  const uint64_t gstart = grp == 0 ? 0 : ((grp & 1) ? s1 : s2);
  const unsigned g0 = __shfl_sync(0xffffffffu, gr[0], grp & 31), g1 = __shfl_sync(0xffffffffu, gr[1], grp & 31);
  const unsigned gw = grp < 32 ? g0 : g1;
  const int kind = gw & 255, gmask = (gw >> 8) & 255, i = (gw >> 16) & 31, j = (gw >> 24) & 31;
  const uint64_t ni = __shfl_sync(0xffffffffu, cnt_l, i), nj = __shfl_sync(0xffffffffu, cnt_l, j);
  const uint64_t si = __shfl_sync(0xffffffffu, start_l, i), sj = __shfl_sync(0xffffffffu, start_l, j);
  if (lane != 0) return;
  uint64_t gb[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) gb[u] = __ldcg(&Ip->grp_base[grp][u]);
  const uint64_t qt = kind ? __ldcg(&Ip->grp_qtiles[grp]) : 1;
  const uint64_t within = local - gstart;
  P.inst = b;
  P.k = k;
  P.T = T;
  P.TP = TP;
  P.half = T / 2;
  P.stride = stride;
  P.mode = mode;
  P.exact = exact;
  P.otf = otf;
  P.split = split;
  P.nolist = nolist;
  P.tab = table;
  P.tmask = tmask;
  // give up early once the table is known to be too small for this level
  P.skip = !otf && ((fails != 0) || (4 * (keys + fresh) > 3 * (tmask + 1)));
  P.kind = kind;
  // operators whose first candidate in this tile comes after the best
  // solution candidate found so far cannot change the result (every
  // candidate before it is still evaluated): they are skipped
  unsigned keep = 0xF;
  int all = gmask;
  if (kind == 0) {
    const uint64_t s0 = within * tq * height, blocks = (ni - s0 + height - 1) >> (7 - split);
    P.nS = ni;
    P.s0 = s0;
    P.srows = rows + si * TP;
    P.nq = (int)(blocks < (uint64_t)tq ? blocks : (uint64_t)tq);
    if (may_skip && best != ~0ULL) {
      keep = 0;
#pragma unroll
      for (int u = 0; u < 4; ++u) keep |= (gb[u] + s0 <= best ? 1u : 0u) << u;
    }
  } else {
    const int qleft = (i == j) || (ni <= nj);
    const uint64_t nS = qleft ? nj : ni, nQ = qleft ? ni : nj;
    uint64_t sq, qr;
    divmod64(within, qt, sq, qr);
    const uint64_t s0 = sq * height, q0 = qr * tq;
    P.qleft = qleft;
    P.nS = nS;
    P.nQ = nQ;
    P.s0 = s0;
    P.q0 = q0;
    P.srows = rows + (qleft ? sj : si) * TP;
    P.qrows = rows + ((qleft ? si : sj) + q0) * TP;
    P.nq = (int)(nQ - q0 < (uint64_t)tq ? nQ - q0 : (uint64_t)tq);
    // the U bits by the staged row's side (staged U stream, stream U staged)
    // rather than by level
    if (!qleft) {
      all = (gmask & 3) | ((gmask & 4) << 1) | ((gmask & 8) >> 1);
      const uint64_t x = gb[2];
      gb[2] = gb[3];
      gb[3] = x;
    }
    if (may_skip && best != ~0ULL) {
      const uint64_t qs = q0 * nS + s0, sm = s0 * nQ + q0, ab = qleft ? qs : sm;
      keep = (gb[0] + ab <= best ? 1u : 0u) | (gb[1] + ab <= best ? 2u : 0u) | (gb[2] + qs <= best ? 4u : 0u) |
             (gb[3] + sm <= best ? 8u : 0u);
    }
  }
#pragma unroll
  for (int u = 0; u < 4; ++u) P.gb[u] = gb[u];
  P.mask = all & keep;
  if (P.mask != all) *(volatile int*)&Ip->p1_masked = 1;
}

// CTA bid of nb: its first tile is tile bid, the later ones come by ticket.
__device__ void ph_p1(const BatchDev& B, unsigned bid, unsigned nb, unsigned long long total) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ TileSh P;
  __shared__ WarpIns s_ins[kTS / 32];
  __shared__ unsigned long long s_red[3][kTS / 32], s_next;
  InsState S{&s_ins[threadIdx.x >> 5], nullptr, 0, 0, 0, false};
  QKey* sK = reinterpret_cast<QKey*>(smem);
  QWord* sQ = reinterpret_cast<QWord*>(smem) + kTQ;
  int prev = -1;   // the instance whose part of P is loaded
  for (unsigned long long tile = bid; tile < total;) {
    const int b = find_owner(B.p1_prefix, B.ninst, tile);
    InstDev& I = B.inst[b];
    if (threadIdx.x < 32) p1_setup(&I, b, tile - B.p1_prefix[b], P);
    else if (b != prev) p1_instance(I, P, 32);
    prev = b;
    __syncthreads();
    // (the next ticket comes back while this tile is worked on)
    unsigned long long next = ~0ULL;
    if (threadIdx.x == 0 && total > nb) next = nb + atomicAdd(B.tickets, 1ULL);
    P1Count cnt{0, 0, ~0ULL};
    // a tile whose every operator is skipped has nothing to do
    const bool idle = P.skip || (!P.otf && P.mask == 0);
    S.list = !P.nolist;
    S.tab = P.tab;
    S.mask = P.tmask;
    if (!idle && P.kind == 1) {
      p1_stage(P, sQ, sK);
      __syncthreads();
    }
    const uint64_t* rows = P.srows;
    if (!idle && P.otf) {
      p1_solutions(P, rows, sQ, cnt);
    } else if (!idle) {
      // a unary tile's rows, kTS (>> split) a step, are one block of the level cache, read
      // once: the next step's are on their way to the L2 during this one
      const int split = P.split;
      const uint64_t height = kTS >> split;
      auto ahead = [&](uint64_t at) {
        if (threadIdx.x || at >= P.nS) return;
        const uint64_t n = P.nS - at < height ? P.nS - at : height;
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;\n" ::"l"(rows + at * P.TP),
                     "r"((unsigned)(n * P.TP * 8)));
      };
      if (P.kind == 0 || P.q0 == 0) ahead(P.s0);
      uint64_t a = P.s0 + (threadIdx.x >> split);
      const uint64_t* row = rows + (a < P.nS ? a : P.nS - 1) * P.TP;
      KeyAcc sk{0, 0};
      if (P.kind && P.mode != KEY_HASH && !split)
        sk = P.mode == KEY_SAMPLED ? row_bits<KEY_SAMPLED>(P, row) : row_bits<KEY_CONCAT>(P, row);
      const bool one = P.mask == 1;
      for (int q = 0; q < P.nq;) {
        int done = 1;
        Cands C;
        C.ok = 0;
        if (P.kind == 0) {
          a = P.s0 + (uint64_t)q * height + (threadIdx.x >> split);
          row = rows + (a < P.nS ? a : P.nS - 1) * P.TP;
          if (q + 1 < P.nq) ahead(P.s0 + (uint64_t)(q + 1) * height);
          if (!split) switch (P.mode) {
            case KEY_HASH: one ? p1_unary<KEY_HASH, 1>(P, row, a, C, cnt) : p1_unary<KEY_HASH, 4>(P, row, a, C, cnt); break;
            case KEY_SAMPLED:
              one ? p1_unary<KEY_SAMPLED, 1>(P, row, a, C, cnt) : p1_unary<KEY_SAMPLED, 4>(P, row, a, C, cnt);
              break;
            default: one ? p1_unary<KEY_CONCAT, 1>(P, row, a, C, cnt) : p1_unary<KEY_CONCAT, 4>(P, row, a, C, cnt);
          }
          else if (P.mode == KEY_HASH) p1_unary_split<KEY_HASH>(P, row, a, C, cnt);
          else p1_unary_split<KEY_CONCAT>(P, row, a, C, cnt);
        } else if (!split) {
          switch (P.mode) {
            case KEY_HASH: done = p1_pair<KEY_HASH>(P, row, sk, sQ, sK, q, C, cnt); break;
            case KEY_SAMPLED: done = p1_pair<KEY_SAMPLED>(P, row, sk, sQ, sK, q, C, cnt); break;
            default: done = p1_pair<KEY_CONCAT>(P, row, sk, sQ, sK, q, C, cnt);
          }
        } else {
          const QWord* qw = sQ + q * P.TP;
          if (P.mode == KEY_HASH) p1_pair_split<KEY_HASH>(P, row, qw, P.q0 + q, a, C, cnt);
          else p1_pair_split<KEY_CONCAT>(P, row, qw, P.q0 + q, a, C, cnt);
        }
        q += done;
        // two candidates at a time, so that the queue stays short (the drain's
        // code is there once; the last drain of the tile empties the queue)
#pragma unroll 1
        for (int r = 0; r < 2; ++r) {
#pragma unroll
          for (int j = 0; j < 2; ++j) push_key(S, (C.ok >> j) & 1u, C.h[j], C.l[j], pay_of(P.k, C.g[j]));
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            C.h[j] = C.h[2 + j];
            C.l[j] = C.l[2 + j];
            C.g[j] = C.g[2 + j];
          }
          C.ok >>= 2;
          drain_queue(I, S, q < P.nq || r == 0 ? 32 * kProbeKeys : 1, cnt);
        }
      }
      if (S.nl) flush_list(I, S, S.nl);
    }
    // per-tile counter flush: warp reductions, then one atomic per counter
    cnt.fresh = warp_sum(cnt.fresh);
    cnt.fail = warp_sum(cnt.fail);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long y = __shfl_down_sync(0xffffffffu, cnt.sol, o);
      cnt.sol = y < cnt.sol ? y : cnt.sol;
    }
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 0) {
      s_red[0][wid] = cnt.sol;
      s_red[1][wid] = cnt.fresh;
      s_red[2][wid] = cnt.fail;
    }
    if (threadIdx.x == 0) s_next = next;
    __syncthreads();
    tile = s_next;   // (written again after the next tile's first barrier)
    if (threadIdx.x == 0) {
      unsigned long long m = ~0ULL, f = 0, x = 0;
      for (int w = 0; w < kTS / 32; ++w) {
        m = s_red[0][w] < m ? s_red[0][w] : m;
        f += s_red[1][w];
        x += s_red[2][w];
      }
      if (m != ~0ULL) atomicMin(&I.best_cand, m);
      if (f) atomicAdd(&I.n_new, f);
      if (P.skip) x += 1;
      if (x) atomicAdd(&I.probe_fail, x);
    }
    // (thread 0 is of the warp that sets the next tile up; no other warp reads
    // P or s_red before that tile's first barrier)
  }
}

__global__ void __launch_bounds__(kTS, 4) k_p1(const __grid_constant__ BatchDev B) {
  step_entry();
  // the tuned CTA count of this step and its tiles (read together)
  const unsigned long long cap = ld_now(B.tickets[kTicketP1Blocks]), total = ld_now(B.p1_prefix[B.ninst]);
  const unsigned nb = cap && cap < gridDim.x ? (unsigned)cap : gridDim.x;
  if (blockIdx.x < nb) ph_p1(B, blockIdx.x, nb, total);
}

// ============================================================== table scan
// Owners of the keys first seen at level k: every slot whose payload carries
// level k.  One chunk of scan_slots slots per CTA iteration; an empty slot's
// payload (~0) carries no level <= 32.  One warp per instance also settles
// whether the recorded solution candidate owns its key.

// The table scan's counting mode at a level that has a solution candidate
// after P1.  The fields read are not written during the scan, except no_mask:
// a failed ownership check sets it while other CTAs of a batch still scan the
// instance's chunks.  A first attempt therefore goes by attempt alone (its
// no_mask was 0 when it was planned): it must not change to marking owners
// half-way, since a last level has no compaction to clear the bitmap
// (last_level).  A later attempt may: its bitmap is always compacted.
__device__ __forceinline__ bool below_mode(const InstDev& I) {
  return I.best_cand != ~0ULL && !I.on_the_fly && (I.attempt == 1 || !I.no_mask);
}

// Level max_size of a search (its first attempt): no later level reads its
// rows, so none are listed or written.  Without a solution candidate after P1
// its result is the number of its owners, which is the number of keys P1
// published; with one, the owners below it are counted (below_mode).  A
// failed ownership check or a buffer found too small builds the level again
// in full.  (49 traces, size 9, nothing found: 8.7 M rows of the last level,
// k_emit 3.2 -> 0.4 ms, the scan 0.45 -> 0.1, the solve 5.83 -> 2.9 ms.)
__device__ __forceinline__ bool last_level(const InstDev& I) {
  return I.level == I.max_size && I.attempt == 1 && !I.keep_last && !I.on_the_fly;
}
__device__ __forceinline__ bool last_unsolved(const InstDev& I) { return last_level(I) && I.best_cand == ~0ULL; }

// What the table scan reads of an instance's record (all of it at once; the
// scan itself changes none of it but the no_mask of a failed ownership check,
// see below_mode).
struct ScanView {
  unsigned long long k, best, newlist, tent, tmask;
  uint64_t plan_words, entries, chunk;
  const Slot* table;
  const uint64_t* wins;
  uint32_t* bitmap;
  bool live, tail, runs, last, below, listed;   // live: its buffers are held
};
__device__ __forceinline__ ScanView scan_view(const InstDev& I) {
  const int status = ld_now(I.status), level = ld_now(I.level), max_size = ld_now(I.max_size),
            attempt = ld_now(I.attempt), keep_last = ld_now(I.keep_last), otf = ld_now(I.on_the_fly),
            no_mask = ld_now(I.no_mask), tail = ld_now(I.p1_tail),
            no_list = ld_now(I.no_list);
  ScanView V;
  V.best = ld_now(I.best_cand);
  V.newlist = ld_now(I.n_newlist);
  V.tent = ld_now(I.tent_cap);
  V.tmask = ld_now(I.table_mask);
  V.plan_words = ld_now(I.plan_words);
  V.chunk = ld_now(I.scan_slots);
  V.table = ld_now_ptr(I.table);
  V.wins = ld_now_ptr(I.wins);
  V.bitmap = ld_now_ptr(I.bitmap);
  V.k = (unsigned long long)level;
  V.live = (status == ST_RUNNING) | (status == ST_NEED_MEM);
  V.tail = tail != 0;
  V.runs = (status == ST_RUNNING) & (tail != 0) & (otf == 0);
  V.last = (level == max_size) & (attempt == 1) & (keep_last == 0) & (otf == 0);
  V.below = (V.best != ~0ULL) & (otf == 0) & ((attempt == 1) | (no_mask == 0));
  // on the first attempt, when every new slot is listed, the list is visited;
  // otherwise (a retried level) the whole table
  V.listed = (attempt == 1) & (no_list == 0) & (V.newlist <= V.tent);
  V.entries = V.listed ? V.newlist : V.tmask + 1;
  return V;
}
__device__ __forceinline__ bool last_unsolved(const ScanView& V) { return V.last & (V.best == ~0ULL); }

// Entries s0 .. s1-1 of the scan, by one CTA.
__device__ void scan_chunk(InstDev& I, const ScanView& V, uint64_t s0, uint64_t s1) {
  __shared__ unsigned long long s_w[32], s_b[32];
  // a level with a solution candidate (where it may skip operators) counts
  // the owners below the candidate instead of marking owner bits (V.below): if
  // the candidate owns its key (nearly always, and always with exact keys)
  // that count is all the level needs; if not, the level is built again in
  // full (the ownership check below)
  unsigned long long cnt = 0, nbelow = 0;
  // kScanBatch entries per thread at a time: their list reads, then their
  // payload reads, are in flight together
  for (uint64_t e0 = s0 + threadIdx.x; e0 < s1; e0 += (uint64_t)kScanBatch * blockDim.x) {
    uint64_t sl[kScanBatch];
    unsigned long long pay[kScanBatch];
#pragma unroll
    for (int u = 0; u < kScanBatch; ++u) {
      const uint64_t e = e0 + (uint64_t)u * blockDim.x;
      sl[u] = e < s1 ? (V.listed ? __ldcg(V.wins + e) : e) : ~0ULL;
    }
#pragma unroll
    for (int u = 0; u < kScanBatch; ++u) pay[u] = sl[u] != ~0ULL ? __ldcg(&V.table[sl[u]].pay) : ~0ULL;
#pragma unroll
    for (int u = 0; u < kScanBatch; ++u) {
      if ((pay[u] >> kPayShift) == V.k) {
        const uint64_t g = pay[u] & kIdxMask;
        if (V.below) nbelow += g < V.best ? 1 : 0;
        else atomicOr(V.bitmap + (g >> 5), 1u << (g & 31));
        ++cnt;
      }
    }
  }
  cnt = warp_sum(cnt);
  nbelow = warp_sum(nbelow);
  if ((threadIdx.x & 31) == 0) {
    s_w[threadIdx.x >> 5] = cnt;
    s_b[threadIdx.x >> 5] = nbelow;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long t = 0, tb = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
      t += s_w[w];
      tb += s_b[w];
    }
    if (t) atomicAdd(&I.n_wins, t);
    if (tb) atomicAdd(&I.n_below, tb);
  }
  __syncthreads();
}

// Every instance's scan, chunks of all instances side by side.  COUNT_LAST: a
// last level without a solution candidate needs no scan (the caller takes the
// count of published keys).
template <bool COUNT_LAST>
__device__ void ph_scan_tables(const BatchDev& B, unsigned bid, unsigned nb) {
  const unsigned long long total = B.tscan_prefix[B.ninst];
  for (unsigned long long c = bid; c < total; c += nb) {
    const int b = find_owner(B.tscan_prefix, B.ninst, c);
    InstDev& I = B.inst[b];
    ScanView V = scan_view(I);
    if (COUNT_LAST && last_unsolved(V)) continue;
    if (V.listed) {
      // the list spread over the instance's chunks, at least a thread's entry each
      const uint64_t nc = B.tscan_prefix[b + 1] - B.tscan_prefix[b], each = (V.entries + nc - 1) / nc;
      if (each < V.chunk) V.chunk = (each + blockDim.x - 1) / blockDim.x * blockDim.x;
    }
    const uint64_t s0 = (c - B.tscan_prefix[b]) * V.chunk;
    if (s0 >= V.entries) continue;   // (uniform over the CTA)
    scan_chunk(I, V, s0, s0 + V.chunk < V.entries ? s0 + V.chunk : V.entries);
  }
}

__device__ void ph_settle_solutions(const BatchDev& B, unsigned bid, unsigned nb) {
  // solution candidate ownership (warp per instance)
  const int lane = threadIdx.x & 31;
  const unsigned long long gw = ((unsigned long long)bid * blockDim.x + threadIdx.x) >> 5;
  const unsigned long long nw = ((unsigned long long)nb * blockDim.x) >> 5;
  for (unsigned long long b = gw; b < (unsigned long long)B.ninst; b += nw) {
    InstDev& I = B.inst[b];
    if (I.status != ST_RUNNING || I.best_cand == ~0ULL || !I.p1_tail || I.on_the_fly) continue;
    const int k = I.level;
    const uint64_t g = I.best_cand;
    const Cand cd = decode(I, k, g);
    if (cd.op < 0) continue;
    uint64_t h, l;
    switch (I.key_mode) {
      case KEY_HASH: warp_key<KEY_HASH>(I, cd, lane, h, l); break;
      case KEY_SAMPLED: warp_key<KEY_SAMPLED>(I, cd, lane, h, l); break;
      default: warp_key<KEY_CONCAT>(I, cd, lane, h, l);
    }
    if (lane == 0) {
      const bool counting = below_mode(I);
      if (find_pay(I.table, I.table_mask, h, l) == pay_of(k, g)) {
        I.best_sol = g;
        I.sol_known = 1;
        I.counted_below = counting ? 1 : 0;
      } else if (I.p1_masked || counting) {
        // an earlier candidate of the level shares the first solution's key
        // (a relaxed-key collision) while operators past it were skipped or
        // the owners were only counted: the level is built again in full (the
        // host re-plans it, nothing to grow)
        I.no_mask = 1;
        I.need = 0;
        I.planned = 0;
        I.status = ST_NEED_MEM;
      }
    }
  }
}

__device__ void ph_table_scan(const BatchDev& B, unsigned bid, unsigned nb) {
  ph_scan_tables<false>(B, bid, nb);
  ph_settle_solutions(B, bid, nb);
}

// An instance's part of the check: its level's buffers against its owners (a
// shortfall asks the host for memory before anything of the level is
// written), its row-emission items.  The owners are known after the level's
// last slice of P1 tiles; an earlier slice (n_wins still 0) only stops at a
// failed probe.  A counted last level (last_unsolved) needs neither list nor
// rows, and is held to the same buffers all the same: which searches a budget,
// a request's cap or the static scratch holds stays what it is for a level
// that is written.
__device__ unsigned long long check_level(InstDev& I) {
  // (status, sol_known and n_wins may have been changed by this kernel: from the L2)
  const int status = __ldcg(&I.status), sk = __ldcg(&I.sol_known), k = ld_now(I.level);
  const unsigned long long wins = __ldcg(&I.n_wins), fresh = ld_now(I.n_new), fails = ld_now(I.probe_fail),
                           keys = ld_now(I.keys), cap = ld_now(I.table_mask) + 1, tent = ld_now(I.tent_cap),
                           row_cap = ld_now(I.row_cap), start = ld_now(I.lstart[k]);
  const bool counted = ld_now(I.p1_tail) != 0 && last_unsolved(I);
  if (status != ST_RUNNING) return 0;
  const unsigned long long nw = counted ? fresh : wins;
  int need = 0;
  if (fails != 0 || 4 * (keys + nw) > 3 * cap) { need |= NEED_TABLE; I.need_amount[1] = 4 * (keys + nw) + 4096; }
  if (nw > tent) { need |= NEED_LIST; I.need_amount[2] = nw; }
  if (!sk && start + nw > row_cap) { need |= NEED_ROWS; I.need_amount[3] = start + nw; }
  if (need) {
    I.need = need;
    I.planned = 0;
    I.status = ST_NEED_MEM;
    return 0;
  }
  if (counted) I.n_wins = nw;
  if (counted || sk) return 0;
  int item = kEmitGroup;
  while (item < kEmitItem && nw > (unsigned long long)item * kEmitItemsFrom) item *= 2;
  I.emit_item = item;
  return (nw + item - 1) / item;
}

// The check of few instances (see scan_compacts), by one CTA: their items'
// prefix, and their small levels' owner bitmaps into the owner lists.  The
// bitmap's words are read while thread 0 checks the buffers.  The record of an
// instance that is done, refused or gave way still names buffers that may be
// somebody else's, or unmapped, by now: nothing behind it is read.
__device__ void check_few(const BatchDev& B, const ScanView& solo, unsigned long long* s_w) {
  __shared__ int s_go;
  unsigned long long items = 0;
  for (int b = 0; b < B.ninst; ++b) {
    InstDev& I = B.inst[b];
    const ScanView V = B.ninst == 1 ? solo : scan_view(I);
    const bool small = V.live && V.tail && small_compact(B, V.plan_words);
    uint32_t v[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const uint64_t w = 2 * threadIdx.x + j;
      v[j] = small && w < V.plan_words ? __ldcg(V.bitmap + w) : 0u;
    }
#pragma unroll
    for (int j = 0; j < 2; ++j)
      if (v[j]) V.bitmap[2 * threadIdx.x + j] = 0u;
    if (threadIdx.x == 0) {
      items += check_level(I);
      B.win_prefix[b + 1] = items;
      s_go = small && *(volatile int*)&I.status == ST_RUNNING;
    }
    unsigned long long tot, pos = block_excl_scan(__popc(v[0]) + __popc(v[1]), s_w, tot);   // (barriers)
    if (s_go) {
      uint64_t* wins = const_cast<uint64_t*>(V.wins);
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        for (uint32_t bits = v[j]; bits; bits &= bits - 1)
          wins[pos++] = (2 * threadIdx.x + j) * 32 + __ffs(bits) - 1;
      }
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) B.win_prefix[0] = 0;
}

// Graph solver: the table scan, then the last CTA to finish checks every
// instance's buffers against its owner count (a shortfall asks the host for
// memory before anything of the level is written) and builds the prefix of
// row-emission items over the instances.  CTAs beyond the level's scan chunks
// (but at least one, and enough warps for the per-instance settle) leave at
// once and take no ticket.
__global__ void __launch_bounds__(kScanThreadsCheck) k_table_scan_check(const __grid_constant__ BatchDev B) {
  __shared__ int s_last;
  __shared__ unsigned long long s_w[32], s_carry;
  step_entry();
  const bool few = scan_compacts(B);
  unsigned long long part;
  ScanView solo;   // the record of a single instance, read once
  // chunks of the levels of few instances as they need them: a list of up to
  // kListChunk slots takes one CTA
  auto job = [&](const ScanView& V, uint64_t& chunk) -> uint64_t {
    chunk = V.listed ? kListChunk : V.chunk;
    return V.runs && !last_unsolved(V) ? V.entries : 0;
  };
  uint64_t chunk;
  if (few) {
    part = 1;
    for (int b = 0; b < B.ninst; ++b) {
      const ScanView V = scan_view(B.inst[b]);
      if (b == 0) solo = V;
      const uint64_t n = job(V, chunk), nc = (n + chunk - 1) / chunk;
      part = nc > part ? nc : part;
    }
  } else {
    const unsigned long long chunks = B.tscan_prefix[B.ninst];
    const unsigned long long want = (unsigned long long)(B.ninst + (blockDim.x >> 5) - 1) / (blockDim.x >> 5);
    part = chunks > want ? chunks : want;
    if (part == 0) part = 1;
  }
  if (part > gridDim.x) part = gridDim.x;
  if (blockIdx.x >= part) return;
  bool solved = !few;   // (few: some instance has a solution candidate)
  if (few) {
    for (int b = 0; b < B.ninst; ++b) {
      InstDev& I = B.inst[b];
      const ScanView V = B.ninst == 1 ? solo : scan_view(I);
      solved |= V.best != ~0ULL;
      const uint64_t n = job(V, chunk);
      for (uint64_t s0 = blockIdx.x * chunk; s0 < n; s0 += part * chunk)
        scan_chunk(I, V, s0, s0 + chunk < n ? s0 + chunk : n);
    }
  } else {
    ph_scan_tables<true>(B, blockIdx.x, (unsigned)part);
    ph_settle_solutions(B, blockIdx.x, (unsigned)part);
  }
  __syncthreads();
  if (part > 1) {
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(B.tickets + 1, 1ULL) == part - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
  }
  if (few) {
    // (settled here, not before: every CTA derives part from the records, which
    // a failed ownership check changes)
    if (solved) ph_settle_solutions(B, 0, 1);
    __syncthreads();
    check_few(B, solo, s_w);
    return;
  }
  if (threadIdx.x == 0) s_carry = 0;
  __syncthreads();
  for (int base = 0; base < B.ninst; base += blockDim.x) {
    const int b = base + threadIdx.x;
    const unsigned long long groups = b < B.ninst ? check_level(B.inst[b]) : 0;
    unsigned long long tot;
    const unsigned long long ex = block_excl_scan(groups, s_w, tot);
    if (b < B.ninst) B.win_prefix[b + 1] = s_carry + ex + groups;
    __syncthreads();
    if (threadIdx.x == 0) s_carry += tot;
    __syncthreads();
  }
  if (threadIdx.x == 0) B.win_prefix[0] = 0;
}

// ========================================================== bitmap compaction
// Owner bitmap (bit g = candidate g owns a new key) -> ascending list I.wins.
__device__ void ph_chunk_count(const BatchDev& B, unsigned bid, unsigned nb) {
  __shared__ unsigned long long s_w[32];
  const unsigned long long* prefix = B.chunk_prefix;
  const unsigned long long total = prefix[B.ninst];
  for (unsigned long long c = bid; c < total; c += nb) {
    const int b = find_owner(prefix, B.ninst, c);
    const InstDev& I = B.inst[b];
    const uint64_t words = (I.cands + 31) / 32;
    const uint64_t w0 = (c - prefix[b]) * kChunkWords;
    const uint64_t w1 = (w0 + kChunkWords < words) ? w0 + kChunkWords : words;
    unsigned long long s = 0;
    for (uint64_t w = w0 + threadIdx.x; w < w1; w += blockDim.x) s += __popc(I.bitmap[w]);
    s = warp_sum(s);
    if ((threadIdx.x & 31) == 0) s_w[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
      unsigned long long t = 0;
      for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += s_w[w];
      B.chunk_cnt[c] = (unsigned int)t;
    }
    __syncthreads();
  }
}

// One CTA per instance: buffer checks for the level's new keys, scan of its
// chunk counts.  The last CTA to finish (ticket) builds the owners' prefix
// over instances.
__device__ void ph_chunk_scan(const BatchDev& B, unsigned bid, unsigned nb) {
  __shared__ unsigned long long s_w[32];
  __shared__ int s_last;
  const unsigned long long* prefix = B.chunk_prefix;
  for (int b = bid; b < B.ninst; b += nb) {
    InstDev& I = B.inst[b];
    if (I.status != ST_RUNNING) continue;
    const unsigned long long c0 = prefix[b], nc = prefix[b + 1] - c0;
    unsigned long long running = 0;
    for (unsigned long long base = 0; base < nc; base += blockDim.x) {
      const unsigned long long i = base + threadIdx.x;
      const unsigned long long v = i < nc ? B.chunk_cnt[c0 + i] : 0ULL;
      unsigned long long tot;
      const unsigned long long ex = block_excl_scan(v, s_w, tot);
      if (i < nc) B.chunk_base[c0 + i] = running + ex;
      running += tot;
    }
    if (threadIdx.x == 0) {
      int need = 0;
      const unsigned long long cap = I.table_mask + 1;
      if (I.probe_fail != 0 || 4 * (I.keys + I.n_wins) > 3 * cap) {
        need |= NEED_TABLE;
        I.need_amount[1] = 4 * (I.keys + I.n_wins) + 4096;
      }
      if (running > I.tent_cap) { need |= NEED_LIST; I.need_amount[2] = running; }
      const uint64_t rows = I.lstart[I.level] + running;
      if (!I.sol_known && rows > I.row_cap) { need |= NEED_ROWS; I.need_amount[3] = rows; }
      I.n_wins = running;
      if (need) {
        I.status = ST_NEED_MEM;
        I.need = need;
      }
    }
    __syncthreads();
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned long long t = atomicAdd(B.tickets + 1, 1ULL);
    s_last = (t == nb - 1);
  }
  __syncthreads();
  if (s_last && threadIdx.x == 0) {
    __threadfence();
    B.win_prefix[0] = 0;
    for (int b = 0; b < B.ninst; ++b) {
      const InstDev& I = B.inst[b];
      const bool run = *(volatile const int*)&I.status == ST_RUNNING &&
                       *(volatile const int*)&I.sol_known == 0;
      B.win_prefix[b + 1] = B.win_prefix[b] + (run ? *(volatile const unsigned long long*)&I.n_wins : 0ULL);
    }
  }
}

// Emit set bits of each chunk in order; always clears the chunk's words.
// The chunk is loaded coalesced into shared memory (padded rows), then every
// thread scans its consecutive words.
__device__ void ph_chunk_emit(const BatchDev& B, unsigned bid, unsigned nb) {
  __shared__ unsigned long long s_w[32];
  const int kPer = kChunkWords / blockDim.x;   // consecutive words per thread
  __shared__ uint32_t s_bits[kChunkWords + 256];
  const unsigned long long* prefix = B.chunk_prefix;
  const unsigned long long total = prefix[B.ninst];
  for (unsigned long long c = bid; c < total; c += nb) {
    const int b = find_owner(prefix, B.ninst, c);
    InstDev& I = B.inst[b];
    const uint64_t words = (I.cands + 31) / 32;
    const uint64_t cbeg = (c - prefix[b]) * kChunkWords;
    for (int u = threadIdx.x; u < kChunkWords; u += blockDim.x) {
      const uint64_t w = cbeg + u;
      const uint32_t v = (w < words) ? I.bitmap[w] : 0u;
      s_bits[(u / kPer) * (kPer + 1) + (u % kPer)] = v;
      if (v) I.bitmap[w] = 0u;
    }
    __syncthreads();
    const uint32_t* mine = s_bits + threadIdx.x * (kPer + 1);
    unsigned long long cnt = 0;
    for (int u = 0; u < kPer; ++u) cnt += __popc(mine[u]);
    unsigned long long tot;
    unsigned long long pos = block_excl_scan(cnt, s_w, tot) + B.chunk_base[c];
    if (I.status == ST_RUNNING && cnt) {
      uint64_t* out = I.wins;
      const uint64_t wbeg = cbeg + (uint64_t)threadIdx.x * kPer;
      for (int u = 0; u < kPer; ++u) {
        const uint32_t bits = mine[u];
        if (!bits) continue;
        const uint64_t base = (wbeg + u) * 32;
#pragma unroll
        for (int p = 0; p < 32; ++p)
          if ((bits >> p) & 1u) out[pos++] = base + p;
      }
    }
    __syncthreads();
  }
}

// ================================================================ emit rows
// Warp per winner, lane per trace word (coalesced row reads and writes).
__device__ void ph_emit_rows(const BatchDev& B, unsigned bid, unsigned nb) {
  const unsigned long long total = B.win_prefix[B.ninst];
  const int lane = threadIdx.x & 31;
  const unsigned long long nwarps = ((unsigned long long)nb * blockDim.x) >> 5;
  for (unsigned long long e = ((unsigned long long)bid * blockDim.x + threadIdx.x) >> 5; e < total;
       e += nwarps) {
    const int b = find_owner(B.win_prefix, B.ninst, e);
    InstDev& I = B.inst[b];
    const uint64_t w = e - B.win_prefix[b];
    const int k = I.level;
    const uint64_t g = I.wins[w];
    const Cand c = decode(I, k, g);
    if (c.op < 0) continue;   // (instances whose solution is settled have no winners listed)
    const uint64_t* ra = row_ptr(I, c.la, c.a);
    const uint64_t* rb = (c.op == OP_AND || c.op == OP_OR || c.op == OP_U) ? row_ptr(I, c.lb, c.b) : ra;
    const uint64_t r = I.lstart[k] + w;
    uint64_t* dst = I.rows + r * (uint64_t)I.TP;
    const int T = I.T;
    unsigned miss = 0u;   // emit_miss OR-ed over the words (the row's own and ~ X F G step-0 tests)
    for (int t = lane; t < I.TP; t += 32) {
      uint64_t word = 0;
      if (t < T) {
        word = apply_w(c.op, __ldcg(ra + t), __ldcg(rb + t), I.len[t]);
        miss |= emit_miss(word, len_mask(I.len[t]), is_pos(I, t) ? 1u : 0u);
      }
      dst[t] = word;
    }
    const unsigned m = __reduce_or_sync(0xffffffffu, miss);
    if (lane == 0) {
      I.origin[r] = g;
      if (!(m & 1u)) atomicMin(&I.best_sol, (unsigned long long)g);
      record_unary(I, k, w, ((m >> 4) & 1u) | (m & 0xEu));   // (~ X F G)
    }
  }
}

// ================================================================== finish
// Bookkeeping of the level just built by a RUNNING instance; on a solution,
// the formula is rebuilt from the cache (LTL_BS.cu:561-705).
__device__ void finish_one(InstDev& I) {
  const int k = I.level;
  if (I.on_the_fly) {
    // nothing of the level was stored: its first solving candidate, if any,
    // is the answer (it owns its word: no earlier candidate or level has it)
    I.lcount[k] = 0;
    I.built_cands = I.cands;
    I.built_wins = 0;
    I.built_scanned = 0;
    I.built_sol_known = 1;
    if (I.best_cand != ~0ULL) {
      const uint64_t g = I.best_cand;
      I.lcands[k] = g + 1;
      I.sol_index = g;
      I.res_size = k;
      I.status = ST_FOUND;
      reconstruct(I, k, g);
    } else {
      I.lcands[k] = I.cands;
      I.res_size = k - 1;
      I.status = ST_LIMIT;
    }
    return;
  }
  // the level's figures are read before the record is written (one thread:
  // a load after a store to the record waits for the store)
  const uint64_t cands = I.cands, wins = I.n_wins, newlist = I.n_newlist, tent = I.tent_cap,
                 cap = I.table_mask + 1, best = I.best_sol, keys = I.keys;
  const uint64_t* wlist = I.wins;
  const uint64_t n_below = I.n_below;
  const int no_list = I.no_list;
  const bool counted = last_unsolved(I);
  const int attempt = I.attempt, sol_known = I.sol_known, max_size = I.max_size,
            counted_below = I.counted_below;
  I.built_cands = cands;
  I.built_wins = wins;
  I.built_scanned = counted ? 0 : (attempt == 1 && !no_list && newlist <= tent) ? newlist : cap;
  I.built_sol_known = sol_known || counted;
  I.keys = keys + wins;
  if (best != ~0ULL) {
    const uint64_t g = best;
    uint64_t lo = 0, hi = wins;   // first index with wins[idx] >= g
    if (counted_below) {
      lo = n_below;
    } else {
      while (lo < hi) {
        const uint64_t mid = (lo + hi) >> 1;
        if (wlist[mid] < g) lo = mid + 1; else hi = mid;
      }
    }
    I.lcount[k] = lo + 1;
    I.lcands[k] = g + 1;
    I.sol_index = g;
    I.res_size = k;
    I.status = ST_FOUND;
    reconstruct(I, k, g);
  } else {
    I.lcount[k] = wins;
    I.lcands[k] = cands;
    I.res_size = k;
    if (k >= max_size) I.status = ST_NOT_FOUND;
    else I.level = k + 1;
  }
  I.rows_deferred = 0;   // the next level projects its rows afresh
}

__device__ void ph_finish(const BatchDev& B, unsigned bid, unsigned nb) {
  for (int b = bid * blockDim.x + threadIdx.x; b < B.ninst; b += nb * blockDim.x) {
    InstDev& I = B.inst[b];
    if (I.status == ST_RUNNING) finish_one(I);
    B.status_out[b] = make_int2(I.status, I.need);
  }
}

// ============================================================ level advance
// One CTA.  built != 0: every RUNNING instance whose level was planned (and
// so built by the step that just ran) is finished; then every RUNNING
// instance not yet planned for its current level is planned.  The batch's
// tile and chunk prefixes are rebuilt from the recorded plans, the
// look-back states of k_compact cleared and the work tickets reset.
__global__ void __launch_bounds__(kAdvanceThreads) k_advance(const __grid_constant__ BatchDev B, cudaGraphConditionalHandle handle, int built,
                                                  int loop, unsigned int max_iter) {
  __shared__ int s_run, s_need;
  __shared__ unsigned s_blocks;
  __shared__ unsigned long long s_w3[32][3];
  __shared__ unsigned long long s_carry[3];
  step_entry();
  // A few instances are warp 0's lanes: their prefixes and totals take a few
  // shuffles instead of block scans and barriers (the kernel runs its code once,
  // from a cold instruction cache): an eight-level search 677 -> 670 us.
  const bool few = scan_compacts(B);
  if (few && threadIdx.x >= 32) return;
  if (!few) {
    if (threadIdx.x == 0) {
      s_run = 0;
      s_need = 0;
      s_blocks = 0;
      s_carry[0] = s_carry[1] = s_carry[2] = 0;
    }
    __syncthreads();
  }
  int run = 0, need = 0;
  unsigned blocks = 0;   // CTAs the step's P1 asks for (~0u: every resident CTA)
  unsigned long long nchunks = 0;
  for (int base = 0; base < B.ninst; base += blockDim.x) {
    const int b = base + threadIdx.x;
    unsigned long long tiles = 0, chunks = 0, tchunks = 0;
    if (b < B.ninst) {
      InstDev& I = B.inst[b];
      const int status = ld_now(I.status), planned = ld_now(I.planned), level = ld_now(I.level), tail = ld_now(I.p1_tail);
      if (built && status == ST_RUNNING && planned == level) {
        if (tail) finish_one(I);
        else I.p1_done += I.p1_step;   // a slice of the level's tiles ran
      }
      if (I.status == ST_RUNNING && I.planned != I.level) plan_one(I, few);
      if (I.status == ST_RUNNING) {
        // this step's slice of P1 tiles: all that remain, or the quota's worth
        const unsigned long long left = I.plan_tiles - I.p1_done;
        unsigned long long step = left;
        if (I.p1_quota && I.cands > I.p1_quota) {
          const unsigned long long q = I.p1_quota * I.plan_tiles / I.cands;
          step = q < 1 ? 1 : (q < left ? q : left);
        }
        I.p1_step = step;
        I.p1_tail = step == left;
        tiles = step;
        const unsigned want = I.p1_blocks ? (unsigned)I.p1_blocks : ~0u;
        blocks = want > blocks ? want : blocks;
        if (I.p1_tail) {
          chunks = last_level(I) || small_compact(B, I.plan_words) ? 0 : (I.plan_words + kCompactWords - 1) / kCompactWords;
          tchunks = I.plan_tchunks;
        }
        run = 1;
      }
      need |= (I.status == ST_NEED_MEM);
      B.status_out[b] = make_int2(I.status, I.need);
    }
    if (few) {
      unsigned long long x[3] = {tiles, chunks, tchunks};
#pragma unroll
      for (int o = 1; o < 4; o <<= 1)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const unsigned long long y = __shfl_up_sync(0xffffffffu, x[c], o);
          if ((int)threadIdx.x >= o) x[c] += y;
        }
      if (b < B.ninst) {
        B.p1_prefix[b + 1] = x[0];
        B.chunk_prefix[b + 1] = x[1];
        B.tscan_prefix[b + 1] = x[2];
      }
      nchunks = __shfl_sync(0xffffffffu, x[1], 3);
      break;
    }
    // inclusive prefixes over this block of instances, carried across blocks
    const unsigned long long v[3] = {tiles, chunks, tchunks};
    unsigned long long ex[3], tot[3];
    block_excl_scan3(v, s_w3, ex, tot);
    if (b < B.ninst) {
      B.p1_prefix[b + 1] = s_carry[0] + ex[0] + tiles;
      B.chunk_prefix[b + 1] = s_carry[1] + ex[1] + chunks;
      B.tscan_prefix[b + 1] = s_carry[2] + ex[2] + tchunks;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      s_carry[0] += tot[0];
      s_carry[1] += tot[1];
      s_carry[2] += tot[2];
    }
    __syncthreads();
  }
  if (few) {
    run = __any_sync(0xffffffffu, run);
    need = __any_sync(0xffffffffu, need);
    blocks = __reduce_max_sync(0xffffffffu, blocks);
  } else {
    if (run) atomicOr(&s_run, 1);
    if (need) atomicOr(&s_need, 1);
    if (blocks) atomicMax(&s_blocks, blocks);
    __syncthreads();
    run = s_run;
    need = s_need;
    blocks = s_blocks;
    nchunks = s_carry[1];
  }
  if (threadIdx.x == 0) {
    B.p1_prefix[0] = 0;
    B.chunk_prefix[0] = 0;
    B.tscan_prefix[0] = 0;
    for (int i = 0; i < 4; ++i) B.tickets[i] = 0;
    B.tickets[kTicketP1Blocks] = blocks == ~0u ? 0 : blocks;
  }
  const unsigned stride = few ? 32u : blockDim.x;
  for (unsigned long long c = threadIdx.x; c < nchunks; c += stride) B.chunk_base[c] = 0;
  if (loop && threadIdx.x == 0) {
    // (the launch's leading advance starts the count)
    const unsigned long long it = *B.loop_iter = built ? *B.loop_iter + 1 : 1;
    const bool more = run && !need && it < max_iter;
    cudaGraphSetConditional(handle, more ? 1u : 0u);
  }
}

// ========================================================= ordered compaction
// Owner bitmap -> ascending owner list I.wins, in one pass.  CTAs take chunks
// of kCompactWords bitmap words in ticket order; each counts its owners,
// publishes the count (flag 1) and then its inclusive prefix (flag 2) in
// chunk_base, and finds its exclusive prefix by looking back over the
// preceding chunks of the instance, a warp at a time (decoupled look-back: a
// chunk waits for its predecessors' counts, which are published as soon as
// they are known, never for their prefixes).  Instances that are not RUNNING
// (the table scan's check asked for memory) are skipped; bitmap words are
// cleared in every case.
constexpr unsigned long long kFlagCount = 1ULL << 62, kFlagPrefix = 2ULL << 62;
constexpr unsigned long long kStateMask = (1ULL << 62) - 1;
constexpr long long kLookbackCycles = 2000000000LL;   // ~1 s: a predecessor that never publishes

__global__ void __launch_bounds__(kCompactThreads) k_compact(const __grid_constant__ BatchDev B) {
  __shared__ unsigned long long s_w[32];
  __shared__ unsigned long long s_c, s_prefix;
  __shared__ int s_ok;
  step_entry();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned long long total = B.chunk_prefix[B.ninst];
  if (blockIdx.x >= total) return;   // no chunk for this CTA (small levels)
  for (;;) {
    if (threadIdx.x == 0) s_c = atomicAdd(B.tickets + 2, 1ULL);
    __syncthreads();
    const unsigned long long c = s_c;
    if (c >= total) break;
    const int b = find_owner(B.chunk_prefix, B.ninst, c);
    InstDev& I = B.inst[b];
    const unsigned long long c0 = B.chunk_prefix[b];
    const uint64_t words = (I.cands + 31) / 32;
    const uint64_t w0 = (c - c0) * kCompactWords;
    uint32_t v[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const uint64_t w = w0 + 2 * threadIdx.x + j;
      v[j] = (w < words) ? __ldcg(I.bitmap + w) : 0u;
      if (v[j]) I.bitmap[w] = 0u;
    }
    const unsigned long long cnt = __popc(v[0]) + __popc(v[1]);
    unsigned long long tot;
    const unsigned long long ex = block_excl_scan(cnt, s_w, tot);
    if (threadIdx.x == 0) {
      const int ok = *(volatile int*)&I.status == ST_RUNNING;
      s_ok = ok;
      if (ok && c == c0) {
        atomicExch(B.chunk_base + c, kFlagPrefix | tot);
        s_prefix = 0;
      } else if (ok) {
        atomicExch(B.chunk_base + c, kFlagCount | tot);
      }
    }
    __syncthreads();
    if (s_ok && c != c0 && warp == 0) {
      // look back: lane i reads chunk (p - i); the nearest chunk with a
      // published prefix ends the walk (chunks before the instance's first
      // count as a prefix of 0)
      unsigned long long prefix = 0;
      long long p = (long long)c - 1;
      bool failed = false;
      for (;;) {
        const long long q = p - lane;
        unsigned long long st = kFlagPrefix;
        if (q >= (long long)c0) {
          const long long t0 = clock64();
          st = *(volatile unsigned long long*)(B.chunk_base + q);
          while ((st >> 62) == 0) {
            if (clock64() - t0 > kLookbackCycles) break;
            st = *(volatile unsigned long long*)(B.chunk_base + q);
          }
        }
        if (__any_sync(0xffffffffu, (st >> 62) == 0)) { failed = true; break; }
        const unsigned pm = __ballot_sync(0xffffffffu, (st >> 62) == 2);
        const int stop = pm ? __ffs(pm) - 1 : 31;
        unsigned long long x = lane <= stop ? (st & kStateMask) : 0ULL;
        x = warp_sum(x);
        prefix += __shfl_sync(0xffffffffu, x, 0);
        if (pm) break;
        p -= 32;
      }
      if (lane == 0) {
        if (failed) {
          // a predecessor never published: give up on this instance; the
          // prefix published here keeps successors' writes inside the list
          atomicExch(&I.status, (int)ST_ERROR);
          prefix = 0;
        }
        atomicExch(B.chunk_base + c, kFlagPrefix | (prefix + tot));
        s_prefix = prefix;
      }
    }
    __syncthreads();
    if (s_ok) {
      unsigned long long pos = s_prefix + ex;
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        uint32_t bits = v[j];
        const uint64_t gw = (w0 + 2 * threadIdx.x + j) * 32;
        while (bits) {
          const int bit = __ffs(bits) - 1;
          bits &= bits - 1;
          I.wins[pos++] = gw + bit;
        }
      }
    }
    __syncthreads();
  }
}

// ================================================================ row emission
// Graph solver: the owners' rows appended to the level cache in canonical
// order, solution test (insertInCache LTL_BS.cu:299-329).  Work items are
// kEmitGroup consecutive owners of one instance on small levels, doubled up to
// kEmitItem on larger ones (prefix built by k_table_scan_check, which records
// the choice).  A warp takes an item: each lane decodes one owner (decode_level:
// compares with the plan's block bases); the item's rows are one block of the
// level cache, which the lanes write 16 bytes at a time side by side, whatever
// the rows' pitch, kEmitUnroll pieces of their operand rows in flight.
// Bound by HBM and instruction issue: level 9 of the large instance (24.3 M rows
// of 64 words, about 19 GB) takes 4.5 ms; with a lane per 8-byte word, a row's
// last words on partly idle warps, and the words' tests one by one, 7.65 ms.
constexpr int kEmitUnroll = 4;
constexpr int kEmitThreads = 256;

// The traces as the emission needs them (per warp): length masks and labels
// (3 for a positive trace: its own and the X test's bit).  The padding word's
// entry repeats the last trace's.
struct __align__(16) EmitTraces {
  uint64_t lm[kMaxTraces];
  uint32_t lab[kMaxTraces];
};

__device__ __forceinline__ ulonglong2 emit_words(int op, ulonglong2 l, ulonglong2 r, ulonglong2 lm, uint64_t second) {
  switch (op) {
    case OP_NOT: return make_ulonglong2(~l.x & lm.x, ~l.y & lm.y & second);
    case OP_AND: return make_ulonglong2(l.x & r.x, l.y & r.y);
    case OP_OR: return make_ulonglong2(l.x | r.x, l.y | r.y);
    case OP_X: return make_ulonglong2(l.x >> 1, l.y >> 1);
    case OP_F: return make_ulonglong2(w_fin(l.x), w_fin(l.y));
    case OP_G: return make_ulonglong2(w_glob(l.x, lm.x), w_glob(l.y, lm.y));
    default: return make_ulonglong2(w_until(l.x, r.x), w_until(l.y, r.y));
  }
}

// emit_miss of two words (see there).
__device__ __forceinline__ unsigned emit_test(uint64_t w0, uint64_t w1, ulonglong2 lm, uint2 lab) {
  const unsigned x0 = (unsigned)w0 ^ lab.x, x1 = (unsigned)w1 ^ lab.y;
  const bool l0 = lab.x != 0, l1 = lab.y != 0;
  const bool f = ((w0 != 0) != l0) || ((w1 != 0) != l1);
  const bool g = (((~w0 & lm.x) == 0) != l0) || (((~w1 & lm.y) == 0) != l1);
  return ((x0 | x1) & 3u) | (f ? 4u : 0u) | (g ? 8u : 0u) | ((~(x0 & x1) & 1u) << 4);
}

__global__ void __launch_bounds__(kEmitThreads, 3) k_emit(const __grid_constant__ BatchDev B) {
  __shared__ EmitTraces s_tr[kEmitThreads / 32];
  step_entry();
  const unsigned long long total = B.win_prefix[B.ninst];
  const int lane = threadIdx.x & 31;
  EmitTraces& tr = s_tr[threadIdx.x >> 5];
  int prev = -1;   // the instance tr holds
  const unsigned long long nw = ((unsigned long long)gridDim.x * blockDim.x) >> 5;
  for (unsigned long long item = ((unsigned long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; item < total;
       item += nw) {
    const int b = find_owner(B.win_prefix, B.ninst, item);
    InstDev& I = B.inst[b];
    const int status = ld_now(I.status), k = ld_now(I.level), T = ld_now(I.T), TP = ld_now(I.TP);
    const uint64_t per = (uint64_t)ld_now(I.emit_item), nwin = ld_now(I.n_wins);
    if (status != ST_RUNNING) continue;
    if (b != prev) {
      prev = b;
      __syncwarp();
      for (int t = lane; t < TP; t += 32) {
        const int u = t < T ? t : T - 1;
        tr.lm[t] = len_mask(I.len[u]);
        tr.lab[t] = is_pos(I, u) ? 3u : 0u;
      }
      __syncwarp();
    }
    const uint64_t o0 = (item - B.win_prefix[b]) * per;
    const int cnt = (int)(nwin - o0 < per ? nwin - o0 : per);
    const uint64_t r0 = I.lstart[k] + o0;
    // lane l decodes owner o0 + l
    int op = -1;
    const uint64_t* pa = I.rows;
    const uint64_t* pb = I.rows;
    uint64_t g = 0;
    if (lane < cnt) {
      g = __ldcg(I.wins + o0 + lane);
      const Cand cd = decode_level(I, k, g);
      op = cd.op;
      if (op >= 0) {
        pa = row_ptr(I, cd.la, cd.a);
        pb = (op == OP_AND || op == OP_OR || op == OP_U) ? row_ptr(I, cd.lb, cd.b) : pa;
        I.origin[r0 + lane] = g;
      }
    }
    const bool pairs = __any_sync(0xffffffffu, pb != pa);   // (an item of unary owners reads one operand)
    // the item's rows as 16-byte units, side by side
    const int U = TP / 2, units = cnt * U;
    const unsigned inv = ((1u << 20) + U - 1) / U;   // f / U = f * inv >> 20 for f below 2^11
    ulonglong2* out = reinterpret_cast<ulonglong2*>(I.rows + r0 * (uint64_t)TP);
    unsigned miss = 0u;   // of this lane's owner: emit_miss OR-ed over its words
    for (int f0 = 0; f0 < units; f0 += 32 * kEmitUnroll) {
      ulonglong2 xa[kEmitUnroll], xb[kEmitUnroll];
      int o[kEmitUnroll], un[kEmitUnroll];
#pragma unroll
      for (int u = 0; u < kEmitUnroll; ++u) {
        const int f = f0 + 32 * u + lane, row = (int)(((unsigned)f * inv) >> 20) & 31;
        un[u] = f - row * U;
        const int ro = __shfl_sync(0xffffffffu, op, row);
        o[u] = f < units ? ro : -1;
        const ulonglong2* a = (const ulonglong2*)__shfl_sync(0xffffffffu, (unsigned long long)pa, row);
        xa[u] = xb[u] = make_ulonglong2(0, 0);
        if (o[u] >= 0) xa[u] = __ldg(a + un[u]);
        if (pairs) {
          const ulonglong2* c = (const ulonglong2*)__shfl_sync(0xffffffffu, (unsigned long long)pb, row);
          if (o[u] >= 0) xb[u] = __ldg(c + un[u]);
        }
      }
#pragma unroll
      for (int u = 0; u < kEmitUnroll; ++u) {
        const int f = f0 + 32 * u;
        if (f >= units) break;   // (warp-uniform)
        unsigned m = 0u;
        if (o[u] >= 0) {
          const ulonglong2 lm = reinterpret_cast<const ulonglong2*>(tr.lm)[un[u]];
          const uint2 lab = reinterpret_cast<const uint2*>(tr.lab)[un[u]];
          const bool pad = 2 * un[u] + 1 == T;
          const ulonglong2 w = emit_words(o[u], xa[u], xb[u], lm, pad ? 0ULL : ~0ULL);
          out[f + lane] = w;
          m = emit_test(w.x, pad ? w.x : w.y, lm, lab);
        }
        if (U == 32) {   // a row per step
          m = __reduce_or_sync(0xffffffffu, m);
          if (lane == f >> 5) miss |= m;
        } else {
          // this lane's owner has units lane * U .. + U - 1: the lanes of this step with some of them
          const int lo = lane * U - f, hi = lo + U;
          const unsigned seg = (hi <= 0 || lo >= 32) ? 0u
                               : (hi >= 32 ? ~0u : (1u << hi) - 1u) & (lo <= 0 ? ~0u : ~0u << lo);
#pragma unroll
          for (int j = 0; j < 5; ++j)
            if (__ballot_sync(0xffffffffu, (m >> j) & 1u) & seg) miss |= 1u << j;
        }
      }
    }
    if (lane < cnt && op >= 0) {
      if (!(miss & 1u)) atomicMin(&I.best_sol, (unsigned long long)g);
      record_unary(I, k, o0 + lane, ((miss >> 4) & 1u) | (miss & 0xEu));   // (~ X F G)
    }
  }
}

// ======================================================= persistent solver
// A wait longer than this (in SM clock cycles, ~60 s) is treated as a failed
// barrier: the waiting CTA raises ctl[2] and every CTA leaves the kernel.
constexpr long long kBarrierCycles = 120000000000LL;

__device__ bool grid_sync(unsigned int* ctl, unsigned int nb) {
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    volatile unsigned int* vgen = ctl + 1;
    volatile unsigned int* verr = ctl + 2;
    const unsigned int gen = *vgen;
    __threadfence();
    const unsigned int arrived = atomicAdd(ctl, 1u) + 1u;
    if (arrived == nb) {
      atomicExch(ctl, 0u);     // no CTA arrives again before the generation moves
      __threadfence();
      atomicAdd(ctl + 1, 1u);
    } else {
      const long long t0 = clock64();
      while (*vgen == gen && *verr == 0) {
        if (clock64() - t0 > kBarrierCycles) {
          atomicExch(ctl + 2, 1u);
          break;
        }
        __nanosleep(64);
      }
    }
    __threadfence();
    s_ok = (*verr == 0);
  }
  __syncthreads();
  return s_ok != 0;
}

__global__ void __launch_bounds__(kTS) k_solve(BatchDev* Bp, unsigned int max_steps) {
  const BatchDev B = *Bp;
  unsigned int* ctl = B.ctl;
  const unsigned int bid = blockIdx.x, nb = gridDim.x;
  __shared__ int s_more;
  for (unsigned int it = 0; it < max_steps; ++it) {
    ph_plan(B, bid, nb);
    if (!grid_sync(ctl, nb)) return;
    if (bid == 0 && threadIdx.x == 0) ph_plan_prefix(B);
    if (!grid_sync(ctl, nb)) return;
    ph_p1(B, bid, nb, B.p1_prefix[B.ninst]);
    if (!grid_sync(ctl, nb)) return;
    ph_table_scan(B, bid, nb);
    if (!grid_sync(ctl, nb)) return;
    ph_chunk_count(B, bid, nb);
    if (!grid_sync(ctl, nb)) return;
    ph_chunk_scan(B, bid, nb);
    if (!grid_sync(ctl, nb)) return;
    ph_chunk_emit(B, bid, nb);
    if (!grid_sync(ctl, nb)) return;
    ph_emit_rows(B, bid, nb);
    if (!grid_sync(ctl, nb)) return;
    ph_finish(B, bid, nb);
    if (!grid_sync(ctl, nb)) return;
    if (bid == 0 && threadIdx.x == 0) {
      int run = 0, need = 0;
      for (int b = 0; b < B.ninst; ++b) {
        const int st = B.status_out[b].x;
        run |= (st == ST_RUNNING);
        need |= (st == ST_NEED_MEM);
      }
      atomicExch(ctl + 3, (run && !need) ? 1u : 0u);
      ++(*B.loop_iter);
    }
    if (!grid_sync(ctl, nb)) return;
    if (threadIdx.x == 0) s_more = *(volatile unsigned int*)(ctl + 3);
    __syncthreads();
    if (!s_more) return;
  }
}

// ========================================================= cluster solver
// One thread-block cluster per instance in flight: the cluster's CTAs run the
// level phases over one instance, separated by the hardware cluster barrier;
// each cluster then pulls the next instance from the queue.  A level above
// the instance's promote_above (or a buffer that must grow) stops the instance
// at a level boundary with NEED_MEM; the host continues it on the whole GPU.
__global__ void __launch_bounds__(kTS) k_cluster(ClusterWork W) {
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  const unsigned int rank = cl.block_rank(), csize = cl.num_blocks();
  const unsigned int slot = blockIdx.x / csize;
  BatchDev B = W.slots[slot];
  __shared__ int s_idx;
  for (;;) {
    if (rank == 0 && threadIdx.x == 0) {
      const unsigned int q = atomicAdd(W.next, 1u);
      s_idx = q < (unsigned int)W.n ? W.order[q] : -1;
    }
    cl.sync();
    const int idx = *cl.map_shared_rank(&s_idx, 0);
    cl.sync();   // rank 0 rewrites s_idx only after every CTA has read it
    if (idx < 0) break;
    B.inst = W.insts + idx;
    B.ninst = 1;
    for (int it = 0; it < kMaxSize + 2; ++it) {
      const int st = *(volatile int*)&B.inst->status;
      cl.sync();   // every CTA has read the status before a phase may change it
      if (st != ST_RUNNING) break;
      ph_plan(B, rank, csize);
      cl.sync();
      if (rank == 0 && threadIdx.x == 0) ph_plan_prefix(B);
      cl.sync();
      ph_p1(B, rank, csize, B.p1_prefix[1]);
      cl.sync();
      ph_table_scan(B, rank, csize);
      cl.sync();
      ph_chunk_count(B, rank, csize);
      cl.sync();
      ph_chunk_scan(B, rank, csize);
      cl.sync();
      ph_chunk_emit(B, rank, csize);
      cl.sync();
      ph_emit_rows(B, rank, csize);
      cl.sync();
      ph_finish(B, rank, csize);
      cl.sync();
    }
  }
}

// ==================================================================== fill
// First buffers of new instances (fill set by the host): empty table (every
// word ~0) and clear owner bitmap, every thread of the grid on one instance
// after the other.  A warp reads the records of 32 instances at once, a lane
// each (one after the other, a batch of 256 waited 0.3 ms for its loads).
__global__ void k_fill(const __grid_constant__ BatchDev B) {
  const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const uint64_t nth = (uint64_t)gridDim.x * blockDim.x;
  const int lane = threadIdx.x & 31;
  for (int b0 = 0; b0 < B.ninst; b0 += 32) {
    const int b = b0 + lane;
    bool mine = false;
    unsigned long long table = 0, slots = 0, bitmap = 0, words = 0;
    if (b < B.ninst) {
      const InstDev& I = B.inst[b];
      mine = I.fill && I.status == ST_RUNNING && I.level == 1;
      table = (unsigned long long)I.table;
      slots = I.table_mask + 1;
      bitmap = (unsigned long long)I.bitmap;
      words = I.bitmap_words;
    }
    for (unsigned m = __ballot_sync(0xffffffffu, mine); m; m &= m - 1) {
      const int j = __ffs(m) - 1;
      ulonglong2* tab = (ulonglong2*)__shfl_sync(0xffffffffu, table, j);
      const uint64_t nt = __shfl_sync(0xffffffffu, slots, j) * (sizeof(Slot) / sizeof(ulonglong2));
      uint32_t* bits = (uint32_t*)__shfl_sync(0xffffffffu, bitmap, j);
      const uint64_t nb = __shfl_sync(0xffffffffu, words, j);
      for (uint64_t x = tid; x < nt; x += nth) tab[x] = make_ulonglong2(~0ULL, ~0ULL);
      for (uint64_t x = tid; x < nb; x += nth) bits[x] = 0u;
    }
  }
}

// ==================================================================== init
// Level 1: every proposition is a row (duplicates included); its key enters
// the set; propositions are tested as size-1 solutions in order
// (LTL_BS.cu:1127-1163, hashSetsInitialisation 136-160).  A warp per
// proposition, a lane per trace word: a thread per proposition walked its
// row word by word, one load after another (6.1 us against 4.9 for a few short
// traces, 45 against 16 for 128).
__global__ void k_init(const __grid_constant__ BatchDev B) {
  __shared__ unsigned long long s_first;
  __shared__ unsigned long long s_new;
  for (int b = blockIdx.x; b < B.ninst; b += gridDim.x) {
    InstDev& I = B.inst[b];
    if (I.status != ST_RUNNING || I.level != 1) continue;
    if (threadIdx.x == 0) {
      s_first = ~0ULL;
      s_new = 0;
      for (int o = 0; o < 4; ++o) I.uhit[atom_level(I)][o] = 0u;
    }
    const bool staged = I.atoms_staged;
    if (staged && !B.atoms) {   // (never: the host uploads them before this launch)
      __syncthreads();
      if (threadIdx.x == 0) I.status = ST_ERROR;
      continue;
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, T = I.T, TP = I.TP, half = T / 2, mode = I.key_mode;
    for (int v = threadIdx.x >> 5; v < I.A; v += blockDim.x >> 5) {
      uint64_t* row = I.rows + (uint64_t)v * TP;
      const uint64_t* from = staged ? B.atoms + I.atom_off + (uint64_t)v * TP : row;
      KeyAcc k;
      key_init(k);
      bool sol = true;
      unsigned miss = 0u;
      for (int t = lane; t < TP; t += 32) {
        const uint64_t w = from[t];
        if (staged) row[t] = w;
        if (t >= T) continue;
        const int L = I.len[t];
        const unsigned lab = is_pos(I, t) ? 1u : 0u;
        sol = sol && (((w & 1ULL) != 0) == (lab != 0));
        miss |= unary_miss(w, len_mask(L), lab);
        if (mode == KEY_HASH) key_word<KEY_HASH>(k, w, t, half, 0, 0, 0, 0);
        else if (mode == KEY_SAMPLED) key_word<KEY_SAMPLED>(k, w, t, half, I.off[t], I.width[t], I.stride1, L);
        else key_word<KEY_CONCAT>(k, w, t, half, I.off[t], I.width[t], 0, L);
      }
      sol = __all_sync(0xffffffffu, sol);
      miss = __reduce_or_sync(0xffffffffu, miss);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        k.a0 ^= __shfl_xor_sync(0xffffffffu, k.a0, o);
        k.a1 ^= __shfl_xor_sync(0xffffffffu, k.a1, o);
      }
      if (lane == 0) {
        uint64_t h, l;
        if (mode == KEY_HASH) key_final<KEY_HASH>(k, h, l);
        else key_final<KEY_CONCAT>(k, h, l);   // (the bit-field modes end alike)
        int isnew = 0;
        uint64_t idx = slot_hash(h, l) & I.table_mask;
        const int r = insert_min(I.table, I.table_mask, idx, ld_key(I.table + idx), h, l,
                                 pay_of(atom_level(I), v), isnew);
        if (r < 0) atomicAdd(&I.probe_fail, 1ULL);
        if (isnew) atomicAdd(&s_new, 1ULL);
        I.origin[v] = v;
        if (sol) atomicMin(&s_first, (unsigned long long)v);
        record_unary(I, atom_level(I), (uint64_t)v, miss);
      }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      I.fill = 0;
      // the propositions are the level of their cost c1 (1 with unit costs);
      // the levels below it are empty
      const int c1 = atom_level(I);
      I.keys = s_new;
      for (int k = 0; k <= c1; ++k) {
        I.lstart[k] = 0;
        I.lcount[k] = 0;
        I.lcands[k] = 0;
      }
      I.lcount[c1] = I.A;
      I.lcands[c1] = I.A;
      I.res_size = c1;
      if (I.probe_fail) {
        I.status = ST_ERROR;
      } else if (s_first != ~0ULL) {
        I.lcount[c1] = s_first + 1;
        I.lcands[c1] = s_first + 1;
        I.sol_index = s_first;
        I.rpn[0] = (int16_t)s_first;
        I.rpn_len = 1;
        I.status = ST_FOUND;
      } else if (I.max_size <= c1) {
        I.status = ST_NOT_FOUND;
      } else {
        I.level = c1 + 1;
      }
      B.status_out[b] = make_int2(I.status, I.need);
    }
    __syncthreads();
  }
}

// ================================================================== rehash
__global__ void k_rehash(const Slot* old_tab, unsigned long long old_cap, Slot* new_tab,
                         unsigned long long new_mask, unsigned long long* fail) {
  for (unsigned long long s = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; s < old_cap;
       s += (unsigned long long)gridDim.x * blockDim.x) {
    const Slot o = old_tab[s];
    if (o.h == kEmpty && o.l == kEmpty) continue;
    uint64_t idx = slot_hash(o.h, o.l) & new_mask;
    bool done = false;
    for (int p = 0; p < kMaxProbes && !done; ++p) {
      const Key128 old = atomicCAS(reinterpret_cast<Key128*>(new_tab + idx), Key128{kEmpty, kEmpty},
                                   Key128{o.h, o.l});
      if (old.h == kEmpty && old.l == kEmpty) {
        new_tab[idx].pay = o.pay;
        done = true;
      } else {
        idx = (idx + 1) & new_mask;
      }
    }
    if (!done) atomicAdd(fail, 1ULL);
  }
}

}  // namespace vfb
