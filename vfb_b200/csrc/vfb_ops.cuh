// vfb_ops.cuh -- device building blocks shared by the level-step kernels
// and the persistent and cluster solvers (vfb_kernels.cu): hash-set
// insert/find, candidate decoding, key computation, P1 tile processing,
// scans, formula reconstruction.
#pragma once
#include "vfb_kernels.cuh"

namespace vfb {

// ------------------------------------------------------------------ helpers
// A field of an instance record, loaded where it is written here: the small
// levels' time is chains of such loads, and one that the compiler moves behind
// the branch on another waits for it (0.6 us each).
__device__ __forceinline__ unsigned long long ld_now(const unsigned long long& x) {
  unsigned long long v;
  asm volatile("ld.global.u64 %0, [%1];\n" : "=l"(v) : "l"(&x));
  return v;
}
__device__ __forceinline__ uint64_t ld_now(const uint64_t& x) {
  uint64_t v;
  asm volatile("ld.global.u64 %0, [%1];\n" : "=l"(v) : "l"(&x));
  return v;
}
__device__ __forceinline__ unsigned ld_now(const unsigned& x) {
  unsigned v;
  asm volatile("ld.global.u32 %0, [%1];\n" : "=r"(v) : "l"(&x));
  return v;
}
__device__ __forceinline__ int ld_now(const int& x) {
  int v;
  asm volatile("ld.global.s32 %0, [%1];\n" : "=r"(v) : "l"(&x));
  return v;
}
template <typename T>
__device__ __forceinline__ T* ld_now_ptr(T* const& x) {
  return (T*)ld_now(reinterpret_cast<const unsigned long long&>(x));
}

__device__ __forceinline__ Key128 ld_key(const Slot* s) {
  const ulonglong2 v = __ldcg(reinterpret_cast<const ulonglong2*>(s));
  return Key128{v.x, v.y};
}

__device__ __forceinline__ unsigned long long pay_of(int k, uint64_t g) {
  return ((unsigned long long)k << kPayShift) | (unsigned long long)g;
}

// Lower the key's payload to pay.  Returns 1 when pay is the key's minimum
// after the update (the candidate may own the key), 0 otherwise.  A payload
// equal to pay means the same candidate claimed it in an earlier attempt of
// this level, which still counts as owning.
__device__ __forceinline__ int claim(Slot* s, unsigned long long pay) {
  const unsigned long long cur = __ldcg(&s->pay);
  if (cur < pay) return 0;
  if (cur == pay) return 1;
  const unsigned long long old = atomicMin(&s->pay, pay);
  return old >= pay ? 1 : 0;
}

// Insert-or-find (h,l) starting at slot idx whose key half-words were already
// loaded into cur.  Returns 1/0 as claim(), -1 when the probe limit is hit.
__device__ inline int insert_min(Slot* tab, uint64_t mask, uint64_t& idx, Key128 cur, uint64_t h, uint64_t l,
                          unsigned long long pay, int& isnew) {
  for (int p = 0; p < kMaxProbes; ++p) {
    if (p > 0) cur = ld_key(tab + idx);
    if (cur.h == h && cur.l == l) return claim(tab + idx, pay);
    // A real key never has a half equal to ~0 (normalised away), so a ~0 half
    // is either an empty slot or a key being published: resolve with the CAS.
    if (cur.h == kEmpty || cur.l == kEmpty) {
      const Key128 old = atomicCAS(reinterpret_cast<Key128*>(tab + idx), Key128{kEmpty, kEmpty},
                                   Key128{h, l});
      if (old.h == kEmpty && old.l == kEmpty) {
        // this thread published the key: its payload is still the empty word,
        // so the minimum needs no read first (and its result is not awaited)
        isnew = 1;
        atomicMin(&tab[idx].pay, pay);
        return 1;
      }
      if (old.h == h && old.l == l) return claim(tab + idx, pay);
    }
    idx = (idx + 1) & mask;
  }
  return -1;
}

// Payload of (h,l), or ~0 if the key is absent.
__device__ inline unsigned long long find_pay(const Slot* tab, uint64_t mask, uint64_t h, uint64_t l) {
  uint64_t idx = slot_hash(h, l) & mask;
  for (int p = 0; p < kMaxProbes; ++p) {
    const Key128 cur = ld_key(tab + idx);
    if (cur.h == h && cur.l == l) return __ldcg(&tab[idx].pay);
    if (cur.h == kEmpty && cur.l == kEmpty) return ~0ULL;
    idx = (idx + 1) & mask;
  }
  return ~0ULL;
}

// Largest b with prefix[b] <= x (prefix non-decreasing, prefix[0] = 0 <= x < prefix[n]).
__device__ __forceinline__ int find_owner(const unsigned long long* prefix, int n, unsigned long long x) {
  int lo = 0, hi = n;  // prefix[lo] <= x < prefix[hi]
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (prefix[mid] <= x) lo = mid; else hi = mid;
  }
  return lo;
}

template <typename V>
__device__ __forceinline__ V warp_sum(V v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

// Block-wide exclusive scan of one value per thread (blockDim multiple of 32).
__device__ inline unsigned long long block_excl_scan(unsigned long long v, unsigned long long* s_warp,
                                              unsigned long long& total) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  unsigned long long x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) s_warp[wid] = x;
  __syncthreads();
  if (wid == 0) {
    unsigned long long w = lane < nw ? s_warp[lane] : 0ULL;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    if (lane < nw) s_warp[lane] = w;
  }
  __syncthreads();
  total = s_warp[nw - 1];
  const unsigned long long before = wid > 0 ? s_warp[wid - 1] : 0ULL;
  __syncthreads();
  return before + x - v;
}

// Three exclusive block scans at once (one pass of barriers): v[c] -> the
// sum of v[c] over the threads before this one; total[c] = the block's sum.
__device__ inline void block_excl_scan3(const unsigned long long (&v)[3], unsigned long long (*s_warp)[3],
                                        unsigned long long (&excl)[3], unsigned long long (&total)[3]) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  unsigned long long x[3] = {v[0], v[1], v[2]};
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const unsigned long long y = __shfl_up_sync(0xffffffffu, x[c], o);
      if (lane >= o) x[c] += y;
    }
  }
  if (lane == 31) {
#pragma unroll
    for (int c = 0; c < 3; ++c) s_warp[wid][c] = x[c];
  }
  __syncthreads();
  if (wid == 0) {
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      unsigned long long w = lane < nw ? s_warp[lane][c] : 0ULL;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long y = __shfl_up_sync(0xffffffffu, w, o);
        if (lane >= o) w += y;
      }
      if (lane < nw) s_warp[lane][c] = w;
    }
  }
  __syncthreads();
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    total[c] = s_warp[nw - 1][c];
    excl[c] = (wid > 0 ? s_warp[wid - 1][c] : 0ULL) + x[c] - v[c];
  }
  __syncthreads();
}

__device__ __forceinline__ uint64_t apply_w(int op, uint64_t l, uint64_t r, int L) {
  switch (op) {
    case OP_NOT: return ~l & len_mask(L);
    case OP_AND: return l & r;
    case OP_OR: return l | r;
    case OP_X: return l >> 1;
    case OP_F: return w_fin(l);
    case OP_G: return w_glob(l, len_mask(L));
    default: return w_until(l, r);
  }
}

struct Cand {
  int op, la, lb;
  uint64_t a, b;
};

// q = g / n, r = g % n.  Below 2^52 the quotient comes from one correctly
// rounded double division (off by at most one, corrected from the remainder),
// which is much shorter than the 64-bit integer division sequence.
__device__ __forceinline__ void divmod64(uint64_t g, uint64_t n, uint64_t& q, uint64_t& r) {
  if (g < (1ULL << 52) && n < (1ULL << 52)) {
    uint64_t qq = (uint64_t)((double)g / (double)n);
    long long rr = (long long)(g - qq * n);
    if (rr < 0) { --qq; rr += (long long)n; }
    else if ((uint64_t)rr >= n) { ++qq; rr -= (long long)n; }
    q = qq;
    r = (uint64_t)rr;
  } else {
    q = g / n;
    r = g % n;
  }
}

// Canonical candidate index g of level k -> operator and operands (levels and
// indices within them).  Block order ~ & | X F G U; a unary operator of cost
// c reads level k - c; & and | over splits (i, k - c - i) with i <= k - c - i,
// U over every split; left index major (ltl_nocache.cu:169-224 with unit
// costs, LTL_BS.cu:1226-1488 with the operator costs).
__device__ inline Cand decode(const InstDev& I, int k, uint64_t g) {
  const uint64_t* n = I.lcount;
  Cand c;
  c.lb = 0;
  c.b = 0;
  if (!I.weighted) {
    // unit costs: the size order
    const uint64_t un = n[k - 1];
    if (g < un) { c.op = OP_NOT; c.la = k - 1; c.a = g; return c; }
    g -= un;
    for (int pass = 0; pass < 2; ++pass) {
      for (int i = 1; 2 * i <= k - 1; ++i) {
        const int j = k - 1 - i;
        const uint64_t cnt = n[i] * n[j];
        if (g < cnt) {
          c.op = pass ? OP_OR : OP_AND;
          c.la = i; c.lb = j;
          divmod64(g, n[j], c.a, c.b);
          return c;
        }
        g -= cnt;
      }
    }
    for (int op = OP_X; op <= OP_G; ++op) {
      if (g < un) { c.op = op; c.la = k - 1; c.a = g; return c; }
      g -= un;
    }
    for (int i = 1; i <= k - 2; ++i) {
      const int j = k - 1 - i;
      const uint64_t cnt = n[i] * n[j];
      if (g < cnt) {
        c.op = OP_U; c.la = i; c.lb = j;
        divmod64(g, n[j], c.a, c.b);
        return c;
      }
      g -= cnt;
    }
    c.op = -1;
    c.la = 1;
    c.a = 0;
    return c;
  }
  const int c1 = atom_level(I);
  const int Ln = not_level(I, k);
  if (Ln >= 0) {
    if (g < n[Ln]) { c.op = OP_NOT; c.la = Ln; c.a = g; return c; }
    g -= n[Ln];
  }
  for (int pass = 0; pass < 2; ++pass) {
    const int w = op_cost(I, pass ? OP_OR : OP_AND);
    for (int i = c1; 2 * i <= k - w; ++i) {
      const int j = k - w - i;
      const uint64_t cnt = n[i] * n[j];
      if (g < cnt) {
        c.op = pass ? OP_OR : OP_AND;
        c.la = i; c.lb = j;
        divmod64(g, n[j], c.a, c.b);
        return c;
      }
      g -= cnt;
    }
  }
  for (int op = OP_X; op <= OP_G; ++op) {
    const int L = k - op_cost(I, op);
    if (L < c1) continue;
    if (g < n[L]) { c.op = op; c.la = L; c.a = g; return c; }
    g -= n[L];
  }
  const int w = op_cost(I, OP_U);
  for (int i = c1; k - w - i >= c1; ++i) {
    const int j = k - w - i;
    const uint64_t cnt = n[i] * n[j];
    if (g < cnt) {
      c.op = OP_U; c.la = i; c.lb = j;
      divmod64(g, n[j], c.a, c.b);
      return c;
    }
    g -= cnt;
  }
  c.op = -1;
  c.la = 1;
  c.a = 0;
  return c;
}

// decode() for a candidate of the level being planned or built (k =
// I.level) with unit costs: the block is found by comparing g with the block
// bases the plan recorded (base_not, base_and / base_or by split, base_x,
// base_f, base_g, base_u by split), then one division splits a pair index.
// Same numbering as decode(); weighted levels take decode().
__device__ inline Cand decode_level(const InstDev& I, int k, uint64_t g) {
  if (I.weighted) return decode(I, k, g);
  const uint64_t* n = I.lcount;
  Cand c;
  c.lb = 0;
  c.b = 0;
  const int ns = (k - 1) / 2;   // & and | splits: left sizes 1..ns
  if (g < I.base_x) {
    if (ns == 0 || g < I.base_and[1]) {
      c.op = OP_NOT; c.la = k - 1; c.a = g - I.base_not;
      return c;
    }
    const bool orb = g >= I.base_or[1];
    const uint64_t* base = orb ? I.base_or : I.base_and;
    int i = 1;
    while (i < ns && g >= base[i + 1]) ++i;
    c.op = orb ? OP_OR : OP_AND;
    c.la = i;
    c.lb = k - 1 - i;
    divmod64(g - base[i], n[k - 1 - i], c.a, c.b);
    return c;
  }
  c.la = k - 1;
  if (g < I.base_f) { c.op = OP_X; c.a = g - I.base_x; return c; }
  if (g < I.base_g) { c.op = OP_F; c.a = g - I.base_f; return c; }
  if (k < 3 || g < I.base_u[1]) {
    if (g - I.base_g < n[k - 1]) { c.op = OP_G; c.a = g - I.base_g; return c; }
    c.op = -1; c.la = 1; c.a = 0;
    return c;
  }
  int i = 1;
  while (i < k - 2 && g >= I.base_u[i + 1]) ++i;
  c.op = OP_U;
  c.la = i;
  c.lb = k - 1 - i;
  divmod64(g - I.base_u[i], n[k - 1 - i], c.a, c.b);
  if (c.a >= n[i]) { c.op = -1; c.la = 1; c.a = 0; c.lb = 0; c.b = 0; }
  return c;
}

__device__ __forceinline__ const uint64_t* row_ptr(const InstDev& I, int lvl, uint64_t idx) {
  return I.rows + (I.lstart[lvl] + idx) * (uint64_t)I.TP;
}

// ======================================================================= P1
// Shared per-tile parameters.  s: the stream operand (a row per thread), q:
// the staged operand (up to kTQ rows, read by every thread).
__device__ __forceinline__ bool exact_keys(const InstDev& I) { return I.exact != 0; }

struct __align__(16) TraceSh {
  uint64_t lm;     // length mask
  uint32_t lab, pad;
};
struct TileSh {
  int inst, k, T, TP, half, stride, mode, skip;
  int kind, mask;   // operand group: 0 unary (bits ~ X F G) / 1 binary (bits & | qUs sUq); the
                    // operators it evaluates
  int otf;          // on-the-fly level: solution test only, nothing inserted
  int nolist;       // new slots are not listed (the table scan reads the whole table)
  int exact;        // every bit of every word is in the key (see InstDev::exact)
  int split;        // log2 of the lanes that share a stream row
  uint64_t s0, q0, nS, nQ;
  int nq;           // staged rows of this tile, or blocks of kTS (>> split) stream rows of a unary one
  const uint64_t *srows, *qrows;   // the stream operand's level; this tile's staged rows
  Slot* tab;
  uint64_t tmask;
  int qleft;        // the staged operand is the left operand of & | (its index is the major one)
  uint64_t gb[4];   // candidate index of each operator of mask at rows (0, 0)
  // ---- the instance's part (kept while consecutive tiles are of one instance)
  TraceSh tr[kMaxTraces];    // (the padding word's trace: all zero)
  uint8_t len[kMaxTraces], off[kMaxTraces], wid[kMaxTraces];
  // exact keys: masks over the 126 key bits: every bit; the last step of
  // each trace; its first step; the labels at the first steps
  unsigned long long full[2], last[2], first[2], want[2];
};

// One staged word: the word, the word >> 30 (first xor-shift of the hash), its
// bits reversed (U), and the trace's label.
struct __align__(16) QWord {
  uint64_t w, sh, rev;
  uint32_t lab, pad;
};
// One staged row of keys that are bit fields: the key's bits, and reversed.
struct __align__(16) QKey {
  uint64_t k0, k1, r0, r1;
};
constexpr int kQWordBytes = 32;
static_assert(sizeof(QWord) == kQWordBytes && sizeof(QKey) == kQWordBytes, "");

struct P1Count {
  unsigned long long fresh, fail, sol;   // keys inserted, probe failures, min solution candidate
};

__device__ __forceinline__ uint64_t ld_row1(const uint64_t* p) {
  uint64_t v;
  asm volatile("ld.global.u64 %0, [%1];\n" : "=l"(v) : "l"(p));
  return v;
}
// Two words of a row (rows start on 16-byte boundaries).
__device__ __forceinline__ void ld_row2(const uint64_t* p, uint64_t& a, uint64_t& b) {
  asm volatile("ld.global.v2.u64 {%0, %1}, [%2];\n" : "=l"(a), "=l"(b) : "l"(p));
}

// body(t, a, b) over the words t = 0, 2, .. TP-2 and t+1 of a row in global
// memory (padding words are zero), snap() before word mid (even).  Every lane
// reads its own row; the next four words are loaded before the current four
// are used.  Measured on the large instance (k_p1 per solve, 20.3 ms): rows
// copied into shared memory eight words ahead, coalesced, 24.1 ms (a tenth
// more instructions); 32-byte loads where the pitch allows 21.5 ms; loads six
// or eight words ahead 22.0-22.7 ms.
template <typename F, typename G>
__device__ __forceinline__ void row_pass(const uint64_t* row, int TP, int mid, F&& body, G&& snap) {
  auto fetch = [&](int t, uint64_t (&x)[4]) {   // t a multiple of 4 below TP
    ld_row2(row + t, x[0], x[1]);
    ld_row2(row + (t + 2 < TP ? t + 2 : t), x[2], x[3]);
  };
  uint64_t v[4];
  fetch(0, v);
#pragma unroll 1
  for (int t = 0; t < TP; t += 4) {
    uint64_t n[4];
    fetch(t + 4 < TP ? t + 4 : t, n);
    const int end = t + 4 < TP ? t + 4 : TP;
#pragma unroll 1
    for (int p = t; p < end; p += 2) {
      if (p == mid) snap();
      body(p, v[0], v[1]);
      v[0] = v[2];
      v[1] = v[3];
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) v[u] = n[u];
  }
}

// ------------------------------------------------ P1's inserts, a warp at a time
// Every candidate's key goes through the warp's queue in shared memory, and
// the queue is worked off kProbeKeys keys per lane at a time: their slots'
// loads, then the CAS of the empty ones, are in flight together.  A key whose
// slot holds another key goes back into the queue for the next slot (linear
// probing), so no lane idles while another follows a chain.  (Resolving every
// thread's four keys in turn, each with its own chain, made the warp wait for
// its longest chain four times over: 23.5 against 20.3 ms of k_p1 on the large
// instance.)  The probe code is there once, whatever the operators computed: a
// copy per operator set ran out of instruction cache (34 ms).
struct __align__(16) Pend {
  uint64_t h, l, pay;
  uint64_t at;   // slot to try next; probes made << kProbeShift
};
constexpr int kProbeShift = 48;
constexpr int kProbeKeys = 2;                          // keys per lane and step
constexpr int kPushKeys = 2;                           // keys per lane queued between two drains
constexpr int kPendCap = 32 * (kProbeKeys + kPushKeys);
constexpr int kNewCap = 64;                            // listed slots: below 32, plus 32
struct WarpIns {
  Pend pend[kPendCap];
  uint64_t fresh[kNewCap];   // slots of new keys, written to the level's list 32 at a time
};
// The warp's side of the queue (every lane holds the same counts).
struct InsState {
  WarpIns* w;
  Slot* tab;
  uint64_t mask;   // of the tile's instance
  int np, nl;
  bool list;
};

// Key and payload of a slot, from L2.
struct SlotVal {
  Key128 key;
  unsigned long long pay;
};
__device__ __forceinline__ SlotVal ld_slot(const Slot* s) {
  const ulonglong2 k = __ldcg(reinterpret_cast<const ulonglong2*>(s));
  return SlotVal{Key128{k.x, k.y}, __ldcg(&s->pay)};
}

// CAS (empty -> key) of a slot where p; else {0, 0}.  Predicated rather than
// branched around, so that several are issued before the first is awaited.
__device__ __forceinline__ Key128 cas_key(bool p, Slot* s, uint64_t h, uint64_t l) {
  Key128 old;
  asm volatile(
      "{\n .reg .pred p;\n .reg .b128 e, n, o;\n setp.ne.u32 p, %2, 0;\n mov.b128 e, {%6, %6};\n"
      " mov.b128 n, {%4, %5};\n mov.b128 o, {%7, %7};\n @p atom.relaxed.gpu.global.cas.b128 o, [%3], e, n;\n"
      " mov.b128 {%0, %1}, o;\n}\n"
      : "=l"(old.h), "=l"(old.l)
      : "r"((unsigned)p), "l"(s), "l"(h), "l"(l), "l"((uint64_t)kEmpty), "l"(0ULL)
      : "memory");
  return old;
}
__device__ __forceinline__ void lower_pay(bool p, Slot* s, unsigned long long pay) {
  asm volatile("{\n .reg .pred p;\n setp.ne.u32 p, %0, 0;\n @p red.relaxed.gpu.global.min.u64 [%1], %2;\n}\n"
               ::"r"((unsigned)p), "l"(&s->pay), "l"(pay) : "memory");
}

// Writes n (at most 32) listed slots to the level's list; the rest move up.
__device__ __forceinline__ void flush_list(InstDev& I, InsState& S, int n) {
  const int lane = threadIdx.x & 31;
  __syncwarp();
  unsigned long long base = 0;
  if (lane == 0) base = atomicAdd(&I.n_newlist, (unsigned long long)n);
  const uint64_t v = S.w->fresh[lane], r = S.w->fresh[32 + lane];
  base = __shfl_sync(0xffffffffu, base, 0);
  if (lane < n && base + lane < I.tent_cap) I.wins[base + lane] = v;
  __syncwarp();
  if (n == 32) S.w->fresh[lane] = r;
  __syncwarp();
  S.nl -= n;
}

// Queues this lane's key (ok; whole warps call this), to start at its home slot.
__device__ __forceinline__ void push_key(InsState& S, bool ok, uint64_t h, uint64_t l, unsigned long long pay) {
  const unsigned m = __ballot_sync(0xffffffffu, ok);
  if (ok) {
    const unsigned lt = (1u << (threadIdx.x & 31)) - 1u;
    S.w->pend[S.np + __popc(m & lt)] = Pend{h, l, pay, slot_hash(h, l) & S.mask};
  }
  S.np += __popc(m);
}

// Works the queue off until fewer than `keep` keys are left.
__device__ __forceinline__ void drain_queue(InstDev& I, InsState& S, int keep, P1Count& cnt) {
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  while (S.np >= keep) {
    __syncwarp();
    const int take = S.np < 32 * kProbeKeys ? S.np : 32 * kProbeKeys;
    S.np -= take;
    Pend k[kProbeKeys];
    SlotVal cur[kProbeKeys];
    Slot* sl[kProbeKeys];
#pragma unroll
    for (int j = 0; j < kProbeKeys; ++j) {
      const int e = lane + 32 * j;
      k[j] = S.w->pend[S.np + (e < take ? e : 0)];
      sl[j] = S.tab + (k[j].at & S.mask);
      cur[j] = SlotVal{Key128{k[j].h, k[j].l}, 0};   // (no key: reads as one that needs nothing)
      if (e < take) cur[j] = ld_slot(sl[j]);
    }
    __syncwarp();   // (every entry is read before a push overwrites it)
    // A real key never has a half equal to ~0 (normalised away), so a ~0 half
    // is either an empty slot or a key being published: resolve with the CAS.
    Key128 old[kProbeKeys];
    unsigned tried = 0;
#pragma unroll
    for (int j = 0; j < kProbeKeys; ++j) {
      const bool e = cur[j].key.h == kEmpty || cur[j].key.l == kEmpty;
      tried |= (unsigned)e << j;
      old[j] = cas_key(e, sl[j], k[j].h, k[j].l);
    }
#pragma unroll
    for (int j = 0; j < kProbeKeys; ++j) {
      const bool e = (tried >> j) & 1u;
      const Key128 now = e ? old[j] : cur[j].key;
      const bool fresh = e && now.h == kEmpty && now.l == kEmpty;   // this lane published the key
      const bool same = now.h == k[j].h && now.l == k[j].l;
      // (the payload of a key just published, here or by another lane, is
      // lowered without a read; of one that was there only if this comes first)
      lower_pay(fresh || (same && (e || cur[j].pay > k[j].pay)), sl[j], k[j].pay);
      cnt.fresh += fresh;
      if (S.list) {
        const unsigned m = __ballot_sync(0xffffffffu, fresh);
        if (m) {
          if (fresh) S.w->fresh[S.nl + __popc(m & lt)] = k[j].at & S.mask;
          S.nl += __popc(m);
          if (S.nl >= 32) flush_list(I, S, 32);
        }
      }
      const uint64_t probes = (k[j].at >> kProbeShift) + 1;
      const bool more = !fresh && !same, lost = more && probes >= (uint64_t)kMaxProbes;
      cnt.fail += lost;
      const unsigned m = __ballot_sync(0xffffffffu, more && !lost);
      if (m) {
        if (more && !lost)
          S.w->pend[S.np + __popc(m & lt)] = Pend{k[j].h, k[j].l, k[j].pay, ((k[j].at + 1) & S.mask) | (probes << kProbeShift)};
        S.np += __popc(m);
      }
    }
  }
}

// Solution test accumulators: only bit 0 (step 0) of a word is compared
// with the trace's label, so 32 bits carry the whole test.
__device__ __forceinline__ uint32_t lo32(uint64_t w) { return (uint32_t)w; }

// Step 0 of ~w, X w, F w and G w on one trace word (length mask lm) against
// the trace's label: bit o set (o = ~ X F G) where it differs.  The same
// bits as the P1 tests of ~w & lm, w >> 1, w_fin(w) and w_glob(w, lm); a row
// whose bits stay clear over every trace makes that operator's candidate on
// it a solution.
__device__ __forceinline__ unsigned unary_miss(uint64_t w, uint64_t lm, unsigned lab) {
  const unsigned n0 = (unsigned)(~w & lm) & 1u;
  const unsigned x0 = (unsigned)(w >> 1) & 1u;
  const unsigned f0 = w != 0 ? 1u : 0u;
  const unsigned g0 = ((w & 1ULL) != 0 && (~w & lm) == 0) ? 1u : 0u;
  return (n0 ^ lab) | ((x0 ^ lab) << 1) | ((f0 ^ lab) << 2) | ((g0 ^ lab) << 3);
}

// The step-0 tests of k_emit on one word of a row, trace lengths being at
// least 1 (so ~w passes exactly where w fails, and G w at step 0 is the word
// covering the whole trace): bit 0 = the row's own test missed, bits 1-4 =
// X, F, G, ~ missed.  OR-ed over the words they are the row's miss bits.
__device__ __forceinline__ unsigned emit_miss(uint64_t w, uint64_t lm, unsigned lab) {
  const unsigned x = ((unsigned)w ^ (lab ? 3u : 0u)) & 3u;
  const unsigned nz = w != 0 ? 1u : 0u;
  const unsigned fu = (~w & lm) == 0 ? 1u : 0u;
  return x | ((nz ^ lab) << 2) | ((fu ^ lab) << 3) | ((~x & 1u) << 4);
}

// Records row `row` of level k as the first one found so far whose ~ X F G
// candidates pass the sample, for the operators whose miss bits are clear.
__device__ __forceinline__ void record_unary(InstDev& I, int k, uint64_t row, unsigned miss) {
  if ((miss & 0xFu) == 0xFu || row >= 0xFFFFFFFFull) return;
  const unsigned v = (unsigned)(0xFFFFFFFFull - row);
#pragma unroll
  for (int o = 0; o < 4; ++o)
    if (!((miss >> o) & 1u)) atomicMax(&I.uhit[k][o], v);
}

// ---- keys that hold every bit of every trace (at most 126 bits)
// The key of a candidate follows from its operands' keys: the operators act on
// all traces at once, the trace fields side by side in 128 bits.  A step must
// not reach into the next field: ~ and X mask it off, and U (a carry chain in
// the reversed order, see until_rev) clears the left operand at each trace's
// last step, where U = r whatever the carry.
struct Bits128 {
  uint64_t a, b;   // bits 0-63, 64-127
};
__device__ __forceinline__ Bits128 rev128(Bits128 x) { return Bits128{__brevll(x.b), __brevll(x.a)}; }
// ln: left operand reversed with the last steps cleared; rr: right operand reversed
__device__ __forceinline__ Bits128 until_exact(Bits128 ln, Bits128 rr) {
  const uint64_t x = ln.a | rr.a, y = ln.b | rr.b;
  uint64_t s, t;
  asm("add.cc.u64 %0, %2, %3;\n\taddc.u64 %1, %4, %5;\n" : "=&l"(s), "=l"(t) : "l"(x), "l"(rr.a), "l"(y), "l"(rr.b));
  return rev128(Bits128{rr.a | (ln.a & ~s), rr.b | (ln.b & ~t)});
}
__device__ __forceinline__ void exact_key(const TileSh& P, Bits128 x, uint64_t& h, uint64_t& l, uint32_t& bad) {
  key_final<KEY_CONCAT>(KeyAcc{x.a, x.b}, h, l);
  bad = (((x.a ^ P.want[0]) & P.first[0]) | ((x.b ^ P.want[1]) & P.first[1])) != 0 ? 1u : 0u;
}

// Up to four candidates of a lane, waiting to be queued.
struct Cands {
  uint64_t h[4], l[4], g[4];
  unsigned ok;    // bit j: candidate j is there
};

// Key bits of a row, one thread per row (bit-field modes).
template <int MODE>
__device__ __forceinline__ KeyAcc row_bits(const TileSh& P, const uint64_t* row) {
  KeyAcc k;
  key_init(k);
  auto word = [&](int t, uint64_t w) { key_word<MODE>(k, w, t, 0, P.off[t], P.wid[t], P.stride, P.len[t]); };
  row_pass(row, P.TP, -1, [&](int t, uint64_t a, uint64_t b) {
    word(t, a);
    word(t + 1, b);
  }, [] {});
  return k;
}

// Candidate j of a lane (ok: it is one).  bad: bit 0 is clear when its step-0
// bits match every trace's label.
__device__ __forceinline__ void take_cand(Cands& C, int j, bool ok, uint64_t g, uint32_t bad, P1Count& cnt) {
  C.g[j] = g;
  C.ok |= (unsigned)ok << j;
  if (ok && !(bad & 1u) && g < cnt.sol) cnt.sol = g;
}

// ---- unary tiles: a row per thread (row a of the level), its ~ X F G candidates
// NU: the operators computed, ~ alone (1: every other one lies past the
// level's first solution) or ~ X F G (4; the inserted ones are P.mask).
template <int MODE, int NU>
__device__ __forceinline__ void p1_unary(const TileSh& P, const uint64_t* row, uint64_t a, Cands& C, P1Count& cnt) {
  uint32_t bad[4] = {0, 0, 0, 0};
  if (MODE == KEY_CONCAT && P.exact) {
    const KeyAcc k = row_bits<KEY_CONCAT>(P, row);
    const Bits128 w{k.a0, k.a1}, n{~w.a & P.full[0], ~w.b & P.full[1]};
    exact_key(P, n, C.h[0], C.l[0], bad[0]);
    if (NU == 4) {
      exact_key(P, Bits128{((w.a >> 1) | (w.b << 63)) & ~P.last[0], (w.b >> 1) & ~P.last[1]}, C.h[1], C.l[1], bad[1]);
      // F w = true U w, G w = ~F~w
      const Bits128 p = rev128(Bits128{P.full[0] & ~P.last[0], P.full[1] & ~P.last[1]});
      exact_key(P, until_exact(p, rev128(w)), C.h[2], C.l[2], bad[2]);
      const Bits128 fn = until_exact(p, rev128(n));
      exact_key(P, Bits128{~fn.a & P.full[0], ~fn.b & P.full[1]}, C.h[3], C.l[3], bad[3]);
    }
  } else if (MODE == KEY_HASH) {
    uint64_t acc[NU], hi[NU];
#pragma unroll
    for (int j = 0; j < NU; ++j) acc[j] = hi[j] = 0;
    auto fold = [&](int j, uint64_t w, uint32_t lab) {
      bad[j] |= lo32(w) ^ lab;
      acc[j] ^= splitmix_mul(w ^ (w >> 30));
    };
    auto word = [&](int t, uint64_t w) {
      const TraceSh x = P.tr[t];
      const uint64_t n = ~w & x.lm;
      fold(0, n, x.lab);
      if (NU == 4) {
        fold(1 % NU, w >> 1, x.lab);
        fold(2 % NU, w_fin(w), x.lab);
        fold(3 % NU, w & ~w_fin(n), x.lab);
      }
    };
    auto snap = [&] {
#pragma unroll
      for (int j = 0; j < NU; ++j) hi[j] = acc[j];
    };
    row_pass(row, P.TP, P.half & ~1, [&](int t, uint64_t x, uint64_t y) {
      word(t, x);
      word(t + 1, y);
    }, snap);
    // the words below T/2 fold into h, the others into l: hi is the fold up
    // to the even word below, an odd T/2's last word is folded in once more
    uint64_t all[NU];
#pragma unroll
    for (int j = 0; j < NU; ++j) {
      all[j] = acc[j];
      acc[j] = 0;
    }
    if (P.half & 1) word(P.half - 1, ld_row1(row + P.half - 1));
#pragma unroll
    for (int j = 0; j < NU; ++j) key_final<KEY_HASH>(KeyAcc{all[j] ^ hi[j] ^ acc[j], hi[j] ^ acc[j]}, C.h[j], C.l[j]);
  } else {
    KeyAcc k[NU];
#pragma unroll
    for (int j = 0; j < NU; ++j) key_init(k[j]);
    auto word = [&](int t, uint64_t w) {
      const TraceSh x = P.tr[t];
      const int L = P.len[t], off = P.off[t], wd = P.wid[t];
      auto put = [&](int j, uint64_t v) {
        bad[j] |= lo32(v) ^ x.lab;
        key_word<MODE>(k[j], v, t, 0, off, wd, P.stride, L);
      };
      put(0, ~w & x.lm);
      if (NU == 4) {
        put(1 % NU, w >> 1);
        put(2 % NU, w_fin(w));
        put(3 % NU, w_glob(w, x.lm));
      }
    };
    row_pass(row, P.TP, -1, [&](int t, uint64_t x, uint64_t y) {
      word(t, x);
      word(t + 1, y);
    }, [] {});
#pragma unroll
    for (int j = 0; j < NU; ++j) key_final<MODE>(k[j], C.h[j], C.l[j]);
  }
#pragma unroll
  for (int j = 0; j < NU; ++j) take_cand(C, j, a < P.nS && ((P.mask >> j) & 1), P.gb[j] + a, bad[j], cnt);
}

// ---- binary tiles: a stream row per thread against the staged rows
// KEYS: the operators computed, among & (1), | (2), staged U stream (4),
// stream U staged (8); the inserted ones are P.mask within it.
template <int K>
struct Keys {
  static constexpr int value = K;
};
__host__ __device__ constexpr int key_count(int keys) {
  return (keys & 1) + ((keys >> 1) & 1) + ((keys >> 2) & 1) + ((keys >> 3) & 1);
}

// Candidates j0.. of one pair (in the order of the bits of KEYS).
template <int KEYS>
__device__ __forceinline__ void take_pair(const TileSh& P, uint64_t q, uint64_t s, int j, const uint32_t* bad,
                                          Cands& C, P1Count& cnt) {
  const uint64_t qs = q * P.nS + s, sq = s * P.nQ + q;
  const uint64_t ab = P.qleft ? qs : sq;
  int u = 0;
#pragma unroll
  for (int o = 0; o < 4; ++o) {
    if (!((KEYS >> o) & 1)) continue;
    take_cand(C, j + u, s < P.nS && ((P.mask >> o) & 1), P.gb[o] + (o < 2 ? ab : o == 2 ? qs : sq), bad[u], cnt);
    ++u;
  }
}

// Hash keys.  Bound by instruction issue and the ALU pipe (level 8 of the large
// instance: 5.5 M candidates of 63 words in 0.623 ms, before 1.092 ms; ALU pipe
// 65%): per word, 11 ALU instructions for & or |, 16 for a U, and 6 multiplies
// each.  The first xor-shift of a & b is (a & b) ^ (a >> 30 & b >> 30), so the
// shifted words are made once per row and word, and the reversed words of U
// too; the last xor-shift is taken once per key (splitmix_end).
// QB staged rows at a time: two where only & and | are kept (the same four keys
// as one row with both U), so that the stream row's loads are shared.
template <int KEYS, int QB>
__device__ __forceinline__ void p1_pair_hash(const TileSh& P, const uint64_t* srow, const QWord* qw, uint64_t q,
                                             uint64_t s, Cands& C, P1Count& cnt) {
  constexpr int N = key_count(KEYS);
  uint64_t acc[QB][N], hi[QB][N];
  uint32_t bad[QB][N];
  auto each = [&](auto&& f) {
#pragma unroll
    for (int b = 0; b < QB; ++b)
#pragma unroll
      for (int j = 0; j < N; ++j) f(b, j);
  };
  each([&](int b, int j) {
    acc[b][j] = hi[b][j] = 0;
    bad[b][j] = 0;
  });
  const int TP = P.TP;
  auto word = [&](int t, uint64_t sw) {
    const uint64_t ssh = sw >> 30;
    const uint64_t srev = (KEYS & 12) ? __brevll(sw) : 0ULL;
#pragma unroll
    for (int b = 0; b < QB; ++b) {
      const QWord x = qw[b * TP + t];
      int j = 0;
      if (KEYS & 1) {
        const uint64_t w = sw & x.w;
        bad[b][j] |= lo32(w) ^ x.lab;
        acc[b][j++] ^= splitmix_mul(w ^ (ssh & x.sh));
      }
      if (KEYS & 2) {
        const uint64_t w = sw | x.w;
        bad[b][j] |= lo32(w) ^ x.lab;
        acc[b][j++] ^= splitmix_mul(w ^ (ssh | x.sh));
      }
      if (KEYS & 4) {
        const uint64_t w = __brevll(until_rev(x.rev, srev));
        bad[b][j] |= lo32(w) ^ x.lab;
        acc[b][j++] ^= splitmix_mul(w ^ (w >> 30));
      }
      if (KEYS & 8) {
        const uint64_t w = __brevll(until_rev(srev, x.rev));
        bad[b][j] |= lo32(w) ^ x.lab;
        acc[b][j++] ^= splitmix_mul(w ^ (w >> 30));
      }
    }
  };
  row_pass(srow, TP, P.half & ~1, [&](int t, uint64_t x, uint64_t y) {
    word(t, x);
    word(t + 1, y);
  }, [&] { each([&](int b, int j) { hi[b][j] = acc[b][j]; }); });
  // (h and l as in p1_unary)
  uint64_t all[QB][N];
  each([&](int b, int j) {
    all[b][j] = acc[b][j];
    acc[b][j] = 0;
  });
  if (P.half & 1) word(P.half - 1, ld_row1(srow + P.half - 1));
  each([&](int b, int j) {
    key_final<KEY_HASH>(KeyAcc{all[b][j] ^ hi[b][j] ^ acc[b][j], hi[b][j] ^ acc[b][j]}, C.h[b * N + j], C.l[b * N + j]);
  });
#pragma unroll
  for (int b = 0; b < QB; ++b) take_pair<KEYS>(P, q + b, s, b * N, bad[b], C, cnt);
}

// Bit-field keys.  The key bits of a & b and a | b follow from the operands'
// (fields and samples are taken bit by bit); those of U too when no field is
// cut (exact: the whole candidate then costs a few dozen instructions whatever
// the number of traces), else from U's words.  sk: the stream row's key bits.
template <int MODE, int KEYS>
__device__ __forceinline__ void p1_pair_bits(const TileSh& P, const uint64_t* srow, const KeyAcc& sk, const QWord* qw,
                                             const QKey& x, uint64_t q, uint64_t s, Cands& C, P1Count& cnt) {
  constexpr int N = key_count(KEYS);
  uint32_t bad[N];
  const KeyAcc kA{sk.a0 & x.k0, sk.a1 & x.k1}, kO{sk.a0 | x.k0, sk.a1 | x.k1};
  int j = 0;
  if (MODE == KEY_CONCAT && P.exact) {
    if (KEYS & 1) { exact_key(P, Bits128{kA.a0, kA.a1}, C.h[j], C.l[j], bad[j]); ++j; }
    if (KEYS & 2) { exact_key(P, Bits128{kO.a0, kO.a1}, C.h[j], C.l[j], bad[j]); ++j; }
    if (KEYS & 12) {
      const Bits128 nl = rev128(Bits128{~P.last[0], ~P.last[1]});
      const Bits128 sr = rev128(Bits128{sk.a0, sk.a1}), qr{x.r0, x.r1};
      if (KEYS & 4) {
        exact_key(P, until_exact(Bits128{qr.a & nl.a, qr.b & nl.b}, sr), C.h[j], C.l[j], bad[j]);
        ++j;
      }
      if (KEYS & 8) {
        exact_key(P, until_exact(Bits128{sr.a & nl.a, sr.b & nl.b}, qr), C.h[j], C.l[j], bad[j]);
        ++j;
      }
    }
  } else {
    KeyAcc k[N];
#pragma unroll
    for (int u = 0; u < N; ++u) {
      key_init(k[u]);
      bad[u] = 0;
    }
    auto word = [&](int t, uint64_t sw) {
      const QWord y = qw[t];
      int u = 0;
      if (KEYS & 1) bad[u++] |= lo32(sw & y.w) ^ y.lab;
      if (KEYS & 2) bad[u++] |= lo32(sw | y.w) ^ y.lab;
      if (KEYS & 12) {
        const uint64_t srev = __brevll(sw);
        auto put = [&](uint64_t w) {
          bad[u] |= lo32(w) ^ y.lab;
          key_word<MODE>(k[u++], w, t, 0, P.off[t], P.wid[t], P.stride, P.len[t]);
        };
        if (KEYS & 4) put(__brevll(until_rev(y.rev, srev)));
        if (KEYS & 8) put(__brevll(until_rev(srev, y.rev)));
      }
    };
    row_pass(srow, P.TP, -1, [&](int t, uint64_t a, uint64_t b) {
      word(t, a);
      word(t + 1, b);
    }, [] {});
    if (KEYS & 1) k[j++] = kA;
    if (KEYS & 2) k[j++] = kO;
#pragma unroll
    for (int u = 0; u < N; ++u) key_final<MODE>(k[u], C.h[u], C.l[u]);
  }
  take_pair<KEYS>(P, q, s, 0, bad, C, cnt);
}

// ---- four lanes to a stream row (small levels, keys that need the words)
// A level that does not fill the SMs is bound by one thread's chain over the
// words of its row: a load's latency every four words and some sixty dependent
// instructions a word.  Here lane s of four takes the words 8i + 2s and the
// next one.  Keys are XOR folds (hashes, or bit fields side by side) and the
// step-0 tests ORs, so the lanes' parts
// combine in two exchanges, which leave candidate s in lane s: one key to
// finish and to queue per lane.  128 traces with sampled keys, levels up to
// 72,000 candidates: the solve 778 -> 603 us; 40 traces, hash keys: k_p1 of
// five levels 92 -> 70 us.  Copies for fewer operators, or per bit-field rule,
// only added code: a small level runs its instructions from a cold cache.
// MODE: KEY_HASH, or KEY_CONCAT for either bit-field key.
// ops(t, w, c): the four candidates' words from word t of the row.
template <int MODE, typename F>
__device__ __forceinline__ void fold_split(const TileSh& P, const uint64_t* row, F&& ops, Cands& C, uint32_t& bad) {
  const int sub = threadIdx.x & 3, TP = P.TP, half = P.half;
  KeyAcc k[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) k[j] = KeyAcc{0, 0};
  uint32_t miss = 0;
  int t = 2 * sub;
  uint64_t v[2] = {0, 0};
  if (t < TP) ld_row2(row + t, v[0], v[1]);
#pragma unroll 1
  for (; t < TP; t += 8) {
    uint64_t n[2];
    ld_row2(row + (t + 8 < TP ? t + 8 : t), n[0], n[1]);
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      uint64_t c[4];
      ops(t + u, v[0], c);
      v[0] = v[1];
      const uint32_t lab = P.tr[t + u].lab;
      const uint64_t below = t + u < half ? ~0ULL : 0ULL;   // (the words below T/2 fold into h)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        miss |= ((lo32(c[j]) ^ lab) & 1u) << j;
        if constexpr (MODE == KEY_HASH) {
          const uint64_t x = splitmix_mul(c[j] ^ (c[j] >> 30));
          k[j].a0 ^= x & ~below;
          k[j].a1 ^= x & below;
        } else {
          const int at = P.off[t + u], wd = P.wid[t + u], L = P.len[t + u];
          if (P.mode == KEY_SAMPLED) key_word<KEY_SAMPLED>(k[j], c[j], t + u, 0, at, wd, P.stride, L);
          else key_word<KEY_CONCAT>(k[j], c[j], t + u, 0, at, wd, P.stride, L);
        }
      }
    }
    v[0] = n[0];
    v[1] = n[1];
  }
  // lanes 0, 1 of four keep candidates 0, 1 and get the others' part of them
  // (2, 3 likewise), then each lane its own
  const unsigned full = 0xffffffffu;
  const bool b2 = sub & 2, b1 = sub & 1;
  auto give = [&](bool up, KeyAcc& x, const KeyAcc& y, int o) {   // x: the kept one of the two
    const uint64_t a0 = __shfl_xor_sync(full, up ? x.a0 : y.a0, o), a1 = __shfl_xor_sync(full, up ? x.a1 : y.a1, o);
    x = KeyAcc{(up ? y.a0 : x.a0) ^ a0, (up ? y.a1 : x.a1) ^ a1};
  };
  give(b2, k[0], k[2], 2);
  give(b2, k[1], k[3], 2);
  give(b1, k[0], k[1], 1);
  key_final<MODE>(k[0], C.h[0], C.l[0]);
  miss |= __shfl_xor_sync(full, miss, 1);
  miss |= __shfl_xor_sync(full, miss, 2);
  bad = miss >> sub;
}

// ~ X F G of row a (one variant: a small level's masked operators cost less
// than another copy of the code).
template <int MODE>
__device__ __forceinline__ void p1_unary_split(const TileSh& P, const uint64_t* row, uint64_t a, Cands& C, P1Count& cnt) {
  uint32_t bad;
  fold_split<MODE>(P, row, [&](int t, uint64_t w, uint64_t (&c)[4]) {
    c[0] = ~w & P.tr[t].lm;
    c[1] = w >> 1;
    c[2] = w_fin(w);
    c[3] = w & ~w_fin(c[0]);
  }, C, bad);
  const int o = threadIdx.x & 3;
  take_cand(C, 0, a < P.nS && ((P.mask >> o) & 1), P.gb[o] + a, bad, cnt);
}

// & | qUs sUq of staged row q (words qw) and stream row s.
template <int MODE>
__device__ __forceinline__ void p1_pair_split(const TileSh& P, const uint64_t* row, const QWord* qw, uint64_t q, uint64_t s,
                                              Cands& C, P1Count& cnt) {
  uint32_t bad;
  fold_split<MODE>(P, row, [&](int t, uint64_t w, uint64_t (&c)[4]) {
    const QWord x = qw[t];
    const uint64_t rev = __brevll(w);
    c[0] = w & x.w;
    c[1] = w | x.w;
    c[2] = __brevll(until_rev(x.rev, rev));
    c[3] = __brevll(until_rev(rev, x.rev));
  }, C, bad);
  const int o = threadIdx.x & 3;
  const uint64_t qs = q * P.nS + s, sq = s * P.nQ + q;
  take_cand(C, 0, s < P.nS && ((P.mask >> o) & 1), P.gb[o] + (o == 2 || (o < 2 && P.qleft) ? qs : sq), bad, cnt);
}

// Staged row q of a binary tile (and the next, where two are taken at a time)
// against this thread's stream row; returns the staged rows done.  The
// operators up to the last one kept: & and | always (& alone is computed with
// |: a variant less, and a smaller kernel image measured faster on small
// levels), either U, or both.
template <int MODE>
__device__ __forceinline__ int p1_pair(const TileSh& P, const uint64_t* srow, const KeyAcc& sk, const QWord* sQ,
                                       const QKey* sK, int q, Cands& C, P1Count& cnt) {
  const uint64_t s = P.s0 + threadIdx.x;
  int done = 1;
  auto go = [&](auto keys) {
    constexpr int K = decltype(keys)::value;
    const QWord* qw = sQ + q * P.TP;
    if constexpr (MODE != KEY_HASH) {
      p1_pair_bits<MODE, K>(P, srow, sk, qw, sK[q], P.q0 + q, s, C, cnt);
    } else {
      if (K == 3 && q + 1 < P.nq) {
        p1_pair_hash<K, K == 3 ? 2 : 1>(P, srow, qw, P.q0 + q, s, C, cnt);
        done = 2;
      } else {
        p1_pair_hash<K, 1>(P, srow, qw, P.q0 + q, s, C, cnt);
      }
    }
  };
  switch (P.mask & 12) {
    case 12: go(Keys<15>{}); break;
    case 8: go(Keys<11>{}); break;
    case 4: go(Keys<7>{}); break;
    default: go(Keys<3>{});
  }
  return done;
}

// On-the-fly level (nothing stored): the tile's candidates get the solution
// test alone, step 0 of every trace against its label; no key, no insert.
__device__ inline void p1_solutions(const TileSh& P, const uint64_t* rows, const QWord* sQ, P1Count& cnt) {
  const uint64_t s = P.s0 + threadIdx.x;
  for (int q = 0; q < P.nq; ++q) {
    const uint64_t a = P.kind ? s : s + (uint64_t)q * kTS;
    if (a >= P.nS) return;
    const uint64_t* row = rows + a * P.TP;
    uint32_t bad[4] = {0, 0, 0, 0};
    uint64_t g[4];
    if (P.kind == 0) {
      auto word = [&](int t, uint64_t w) {
        const TraceSh x = P.tr[t];
        bad[0] |= lo32(~w & x.lm) ^ x.lab;
        bad[1] |= lo32(w >> 1) ^ x.lab;
        bad[2] |= lo32(w_fin(w)) ^ x.lab;
        bad[3] |= lo32(w_glob(w, x.lm)) ^ x.lab;
      };
      row_pass(row, P.TP, -1, [&](int t, uint64_t x, uint64_t y) {
        word(t, x);
        word(t + 1, y);
      }, [] {});
#pragma unroll
      for (int j = 0; j < 4; ++j) g[j] = P.gb[j] + a;
    } else {
      const QWord* qw = sQ + q * P.TP;
      auto word = [&](int t, uint64_t sw) {
        const QWord y = qw[t];
        const uint64_t srev = __brevll(sw);
        bad[0] |= lo32(sw & y.w) ^ y.lab;
        bad[1] |= lo32(sw | y.w) ^ y.lab;
        bad[2] |= lo32(__brevll(until_rev(y.rev, srev))) ^ y.lab;
        bad[3] |= lo32(__brevll(until_rev(srev, y.rev))) ^ y.lab;
      };
      row_pass(row, P.TP, -1, [&](int t, uint64_t x, uint64_t y) {
        word(t, x);
        word(t + 1, y);
      }, [] {});
      const uint64_t qs = (P.q0 + q) * P.nS + s, sq = s * P.nQ + P.q0 + q, ab = P.qleft ? qs : sq;
      g[0] = P.gb[0] + ab;
      g[1] = P.gb[1] + ab;
      g[2] = P.gb[2] + qs;
      g[3] = P.gb[3] + sq;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (((P.mask >> j) & 1) && !(bad[j] & 1u) && g[j] < cnt.sol) cnt.sol = g[j];
  }
}

// Warp per candidate, lane per trace word: the two operand rows are read
// coalesced, every lane folds its words into a partial key, and the partial
// keys are combined with XOR shuffles (hash mode XOR-folds by definition; the
// bit fields of the other modes are disjoint, so XOR equals OR).
template <int MODE>
__device__ __forceinline__ void warp_key(const InstDev& I, const Cand& c, int lane, uint64_t& h, uint64_t& l) {
  const uint64_t* ra = row_ptr(I, c.la, c.a);
  const uint64_t* rb = (c.op == OP_AND || c.op == OP_OR || c.op == OP_U) ? row_ptr(I, c.lb, c.b) : ra;
  KeyAcc k;
  key_init(k);
  const int T = I.T, half = T / 2;
  for (int t = lane; t < T; t += 32) {
    const uint64_t w = apply_w(c.op, __ldcg(ra + t), __ldcg(rb + t), I.len[t]);
    key_word<MODE>(k, w, t, half, I.off[t], I.width[t], I.stride1, I.len[t]);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    k.a0 ^= __shfl_xor_sync(0xffffffffu, k.a0, o);
    k.a1 ^= __shfl_xor_sync(0xffffffffu, k.a1, o);
  }
  key_final<MODE>(k, h, l);
}

// RPN of the node (level lvl, candidate g) into I.rpn (postfix).
// RPN of candidate g of level lvl, rebuilt through the operands' canonical
// indices (origin); returns its length (0 if it does not fit cap).
__device__ inline int reconstruct_to(const InstDev& I, int lvl, uint64_t g, int16_t* rpn, int cap) {
  struct Fr { int lvl; uint64_t g; int state; };
  Fr st[2 * kMaxSize + 2];
  int sp = 0, out = 0;
  st[0] = {lvl, g, 0};
  while (sp >= 0) {
    if (out >= cap) return 0;
    Fr& f = st[sp];
    if (f.lvl <= atom_level(I)) {
      rpn[out++] = (int16_t)f.g;
      --sp;
      continue;
    }
    const Cand c = decode(I, f.lvl, f.g);
    if (c.op < 0) return 0;
    const bool bin = (c.op == OP_AND || c.op == OP_OR || c.op == OP_U);
    if (f.state == 0) {
      f.state = 1;
      st[++sp] = {c.la, I.origin[I.lstart[c.la] + c.a], 0};
    } else if (f.state == 1 && bin) {
      f.state = 2;
      st[++sp] = {c.lb, I.origin[I.lstart[c.lb] + c.b], 0};
    } else {
      rpn[out++] = (int16_t)(-(1 + c.op));
      --sp;
    }
  }
  return out;
}

__device__ inline void reconstruct(InstDev& I, int lvl, uint64_t g) {
  I.rpn_len = reconstruct_to(I, lvl, g, I.rpn, kMaxSize);
}

}  // namespace vfb
