// vfb_exhaustive.cu -- cache-free search in formula-number order.
//
// The reference's ltl_nocache (ltl_nocache.cu:319-446) evaluates every
// formula of a size, numbered by numberToFormula (ltl_nocache.cu:169-224) over
// the count matrix of generateMatrix (ltl_nocache.cu:248-287), and keeps any
// solution of the first operator block that has one (a race inside the block).
// Here each thread decodes a formula number and tests the formula trace by
// trace (most formulas fail on the first traces), and lowers the smallest
// solving number with atomicMin, so the host gets the first solution of the
// numbering order.  No deduplication and no hash set: every number is tested.
//
// The words of all formulas of the smallest sizes 1..m (as many as fit
// kExhTableWords words: 8 MB) are written to a table first, so that a larger
// formula is decoded only down to its subformulas of those sizes: a size-9
// formula of three propositions is an operator or two over table entries
// instead of nine nodes, each with its own search through the count matrix and
// its own division.  (Three propositions, ten traces: size 8, 1.18 M formulas,
// 115 -> 48 us; size 9 until its first solution 475 -> 181 us.)
#include "vfb_ops.cuh"

namespace vfb {

// Root of formula number n of size k >= 2 (cnt[s][op] = formulas of size s
// whose root is op, cnt[s][7] = all of size s): its operator, its operands'
// sizes and numbers (left or only one first; ls + rs + 1 = k, rs = 0: unary).
struct ExhRoot {
  int op, ls, rs;
  uint64_t ln, rn;
};
__device__ __forceinline__ ExhRoot exh_root(uint64_t n, int k, const uint64_t (*cnt)[8]) {
  ExhRoot r;
  r.op = 0;
  while (r.op < OP_U && n >= cnt[k][r.op]) n -= cnt[k][r.op++];
  const int sub = k - 1;
  if (r.op == OP_NOT || r.op == OP_X || r.op == OP_F || r.op == OP_G) {
    r.ls = sub;
    r.rs = 0;
    r.ln = n;
    r.rn = 0;
    return r;
  }
  int left = 1;
  while (left < sub - 1 && n >= cnt[left][7] * cnt[sub - left][7]) {
    n -= cnt[left][7] * cnt[sub - left][7];
    ++left;
  }
  r.ls = left;
  r.rs = sub - left;
  divmod64(n, cnt[r.rs][7], r.ln, r.rn);
  return r;
}

// Formula number n of size k in reverse Polish order from the end of tok:
// table entries (>= 0) for subformulas of at most m nodes, else operators
// (-(1 + operator)).  Returns the first token's position.
__device__ __forceinline__ int exh_decode(uint64_t n, int k, const ExhDev& P, const uint64_t (*cnt)[8], int* tok) {
  struct Pend {
    uint64_t n;
    int size;
  };
  Pend st[kMaxSize];
  int sp = 0, at = kMaxSize;
  st[0] = Pend{n, k};
  while (sp >= 0) {
    const Pend e = st[sp--];
    if (e.size <= P.m) {
      tok[--at] = (int)(P.first[e.size] + e.n);
      continue;
    }
    const ExhRoot r = exh_root(e.n, e.size, cnt);
    tok[--at] = -(1 + r.op);
    st[++sp] = Pend{r.ln, r.ls};
    if (r.rs) st[++sp] = Pend{r.rn, r.rs};   // (the right operand's tokens come next before the root)
  }
  return at;
}

// 1 iff the formula holds at step 0 of every positive trace and of no
// negative trace (semantics of evaluateRPN, ltl_nocache.cu:78-161).
__device__ __forceinline__ bool exh_solves(const ExhDev& P, const int* tok, int at) {
  for (int t = 0; t < P.T; ++t) {
    uint64_t stk[kMaxSize];
    int sp = 0;
    const int L = P.len[t];
    const uint64_t* w = P.tab + (size_t)t * P.entries;
    for (int i = at; i < kMaxSize; ++i) {
      const int k = tok[i];
      if (k >= 0) {
        stk[sp++] = __ldg(w + k);
      } else {
        const int op = -k - 1;
        if (op == OP_AND || op == OP_OR || op == OP_U) {
          const uint64_t r = stk[--sp];
          stk[sp - 1] = apply_w(op, stk[sp - 1], r, L);
        } else {
          stk[sp - 1] = apply_w(op, stk[sp - 1], 0, L);
        }
      }
    }
    const uint64_t want = (P.posmask[t >> 6] >> (t & 63)) & 1ULL;
    if ((stk[0] & 1ULL) != want) return false;
  }
  return true;
}

// The count matrix in shared memory; whether a smaller size has a solution
// (best[s]: smallest solving number of size s): nothing is left to find then.
__device__ __forceinline__ bool exh_begin(const ExhDev& P, int k, const unsigned long long* best,
                                          uint64_t (*cnt)[8]) {
  __shared__ int s_done;
  if (threadIdx.x == 0) {
    s_done = 0;
    for (int s = 1; s < k; ++s) s_done |= __ldcg(best + s) != ~0ULL;
  }
  for (int i = threadIdx.x; i < (k + 1) * 8; i += blockDim.x) cnt[i / 8][i % 8] = P.cnt[i / 8][i % 8];
  __syncthreads();
  return !s_done;
}

// Size k <= m: the table's words of every formula of the size, and their
// solution test.
__global__ void __launch_bounds__(256) k_exh_table(const ExhDev* __restrict__ Pp, int k, unsigned long long* best) {
  __shared__ uint64_t s_cnt[kMaxSize + 1][8];
  const ExhDev& P = *Pp;
  if (!exh_begin(P, k, best, s_cnt)) return;
  const uint64_t total = s_cnt[k][7];
  for (uint64_t n = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; n < total; n += (uint64_t)gridDim.x * blockDim.x) {
    ExhRoot r{-1, 0, 0, 0, 0};
    if (k > 1) r = exh_root(n, k, s_cnt);
    const uint64_t a = P.first[r.ls] + r.ln, b = r.rs ? P.first[r.rs] + r.rn : a, o = P.first[k] + n;
    bool sol = true;
    for (int t = 0; t < P.T; ++t) {
      uint64_t* w = P.tab + (size_t)t * P.entries;
      const uint64_t v = k == 1 ? P.words[(size_t)t * P.A + n] : apply_w(r.op, w[a], w[b], P.len[t]);
      w[o] = v;
      sol = sol && (v & 1ULL) == ((P.posmask[t >> 6] >> (t & 63)) & 1ULL);
    }
    if (sol) atomicMin(best + k, (unsigned long long)n);
  }
}

// Size k > m: formula numbers [lo, hi) are evaluated and the smallest solving
// number lowers best[k].
__global__ void __launch_bounds__(256) k_exhaustive(const ExhDev* __restrict__ Pp, int k, unsigned long long lo,
                                                    unsigned long long hi, unsigned long long* best) {
  __shared__ uint64_t s_cnt[kMaxSize + 1][8];
  const ExhDev& P = *Pp;
  if (!exh_begin(P, k, best, s_cnt)) return;
  const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
  unsigned long long seen = *(volatile unsigned long long*)(best + k);
  int tok[kMaxSize];
  unsigned it = 0;
  for (unsigned long long n = lo + (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; n < hi; n += stride) {
    // a smaller solving number already found: nothing left to gain here
    if ((++it & 31u) == 0) seen = *(volatile unsigned long long*)(best + k);
    if (n >= seen) break;
    const int at = exh_decode(n, k, P, s_cnt, tok);
    if (exh_solves(P, tok, at)) atomicMin(best + k, n);
  }
}

}  // namespace vfb
