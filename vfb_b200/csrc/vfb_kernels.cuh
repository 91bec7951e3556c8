// vfb_kernels.cuh -- kernel entry points of the level step (see vfb_kernels.cu).
#pragma once
#include "vfb_device.cuh"

namespace vfb {

constexpr int kChunkWords = 4096;     // bitmap words per compaction chunk (131072 bits)
constexpr int kScanSlots = 1024;      // hash-set slots per table-scan chunk (at least; more on
                                      // larger tables, see scan_slots)
constexpr int kScanThreadsCheck = 256; // threads per k_table_scan_check CTA
constexpr uint64_t kListChunk = 1024; // listed slots per table-scan chunk when few instances run
constexpr int kScanBatch = 8;         // table-scan entries a thread reads at a time
constexpr int kCompactWords = 512;    // owner-bitmap words per k_compact chunk (16384 candidates)
constexpr int kCompactThreads = 256;  // threads per k_compact CTA (two bitmap words each)
// k_advance threads at most (it loops over larger batches): few enough that
// the one-thread plan and finish keep their state in registers
constexpr int kAdvanceThreads = 256;
constexpr int kTickets = 8;            // words of BatchDev::tickets
constexpr int kTicketP1Blocks = 4;     // tickets[4]: CTAs the step's k_p1 runs (0: all), set by k_advance
constexpr int kEmitGroup = 4;         // owners per k_emit work item at least (doubled as the level grows)
constexpr int kEmitItem = 32;         // owners per k_emit work item at most (one warp; a lane
                                      // decodes each); small levels take as few as kEmitGroup so
                                      // that their owners still spread over many warps
constexpr unsigned long long kEmitItemsFrom = 4736;   // items (32 warps an SM) from which they are doubled

// Staged rows of a P1 tile at most, and the dynamic shared memory of k_p1 for
// rows of up to TP words: the staged rows' key bits and words (32 bytes each,
// see QWord and QKey), at most 9 KB, so that the registers and not the shared
// memory bound the CTAs of an SM.
__host__ __device__ constexpr int p1_rows_max(int TP) { return TP > 64 ? 2 : TP > 32 ? 4 : TP > 16 ? 8 : kTQ; }
__host__ __device__ constexpr int p1_smem_bytes(int TP) { return 32 * (kTQ + (TP > 16 ? 264 : kTQ * TP)); }
static_assert(p1_rows_max(128) * 128 <= 264 && p1_rows_max(64) * 64 <= 264 && p1_rows_max(32) * 32 <= 264, "");

// Global batch descriptor, passed by value (a load less at the head of every
// kernel); the instance records it points to stay in place when buffers grow,
// and a captured launch sequence is built again when the workspace moves.
struct BatchDev {
  InstDev* inst;
  int ninst;
  int pad;
  unsigned long long* p1_prefix;        // [ninst+1] P1 tiles
  unsigned long long* chunk_prefix;     // [ninst+1] owner-bitmap chunks
  unsigned long long* tscan_prefix;     // [ninst+1] table-scan chunks
  unsigned long long* win_prefix;       // [ninst+1] owners of new keys (ph_emit_rows), or
                                        // row-emission groups (k_emit)
  unsigned int* chunk_cnt;              // [chunk_cap]
  unsigned long long* chunk_base;       // [chunk_cap] chunk offsets (ph_chunk_*), or the
                                        // look-back states of k_compact (flag << 62 | count)
  unsigned long long chunk_cap;
  unsigned long long* tickets;          // [kTickets]: P1 work ticket, scan done counter,
                                        // compaction ticket, (unused), P1 CTAs of the step
  int2* status_out;                     // [ninst] (status, need) mirror for the host
  unsigned long long* loop_iter;        // level steps run by the current device-side loop
  const uint64_t* atoms;                // proposition rows of the call's new instances (one upload),
                                        // copied into each level cache by k_init
  unsigned int* ctl;                    // persistent solver: [0] barrier arrivals, [1] barrier
                                        // generation, [2] error, [3] continue flag
};

// Level step of the graph solver: k_p1, k_table_scan_check, k_compact,
// k_emit, k_advance (k_advance also runs once, with built = 0, before the
// first step of a launch).  k_table_scan_check adds the buffer checks to the
// table scan; k_compact replaces the chunk count, scan and emission with one
// ordered pass (decoupled look-back over the chunks); k_advance does the
// finish, the plan and the loop control.  With loop != 0 it sets the graph's while
// condition: some instance RUNNING, none waiting for memory, fewer than
// max_iter steps.
__global__ void k_advance(const __grid_constant__ BatchDev B, cudaGraphConditionalHandle handle, int built, int loop,
                          unsigned int max_iter);
__global__ void k_table_scan_check(const __grid_constant__ BatchDev B);
__global__ void k_compact(const __grid_constant__ BatchDev B);
__global__ void k_emit(const __grid_constant__ BatchDev B);

__global__ void k_p1(const __grid_constant__ BatchDev B);

// Persistent solver: the whole level loop in one cooperative launch (all CTAs
// co-resident), the phases above separated by a bounded grid barrier.  Runs at
// most max_steps levels; stops early when no instance is RUNNING or one needs
// memory.  ctl[2] != 0 afterwards means a barrier timed out.
__global__ void k_solve(BatchDev* B, unsigned int max_steps);

// Cluster solver work list: slots[c] is cluster c's private workspace (one
// instance at a time), insts the instance records, order the queue of record
// indices, next its head.
struct ClusterWork {
  BatchDev* slots;
  InstDev* insts;
  const int* order;
  int n;
  unsigned int* next;
};
__global__ void k_cluster(ClusterWork W);

// Cache-free search (vfb_exhaustive.cu): the instance, the count matrix of
// the formula numbering, and the table of the words of all formulas of sizes
// 1..m: tab[t * entries + first[s] + n] = formula n of size s on trace t.
constexpr uint64_t kExhTableWords = 1ull << 20;
struct ExhDev {
  int A, T, m;
  uint64_t entries;
  uint64_t* tab;
  uint64_t first[kMaxSize + 1];    // first[0] unused
  uint64_t cnt[kMaxSize + 1][8];   // formulas per size and root operator (7: all of the size)
  uint64_t posmask[2];             // bit t: trace t is positive
  uint8_t len[kMaxTraces];
  uint64_t words[kMaxTraces * 64]; // words[t * A + v]: proposition v on trace t
};
__global__ void k_exh_table(const ExhDev* P, int k, unsigned long long* best);
__global__ void k_exhaustive(const ExhDev* P, int k, unsigned long long lo, unsigned long long hi,
                             unsigned long long* best);

// BS stage (vfb_bs.cu): words of the cache rows and of their ~ & |
// combinations, in a slot table of their own.
constexpr int kBsChunkWords = 1024;   // bitmap words per compaction chunk of the BS stage
struct BsDev {
  const uint64_t* rows;            // the instance's level cache (pitch TP)
  int T, TP;
  uint64_t full, target;           // T low bits; the positive traces' bits
  Slot* tab;
  unsigned long long mask;         // table capacity - 1
  uint64_t* vals;                  // entries: words, in canonical order
  uint64_t* org;                   // entries: cache row (base) or candidate index
  uint32_t* bitmap;                // owner bits of the size being built
  unsigned long long* counts;      // owners per chunk
  unsigned long long* offs;        // chunk offsets (exclusive prefix of counts)
  unsigned long long* best;        // first solving candidate of the size
  unsigned long long* fail;        // probe failures
  unsigned long long* total;       // owners of the size
  uint64_t st[kMaxSize + 2], cn[kMaxSize + 2];   // first entry and entries of each size
};
struct BsCand {
  int op;
  uint64_t a, b;   // entry indices of the operands
};

// Candidate g of BS size c -> operator and operand entries.
__host__ __device__ inline BsCand bs_decode(const uint64_t* st, const uint64_t* cn, int c, uint64_t g) {
  BsCand r{-1, 0, 0};
  const uint64_t un = cn[c - 1];
  if (g < un) return BsCand{OP_NOT, st[c - 1] + g, 0};
  g -= un;
  for (int pass = 0; pass < 2; ++pass) {
    for (int i = 1; 2 * i <= c - 1; ++i) {
      const int j = c - 1 - i;
      const uint64_t n = cn[i] * cn[j];
      if (g < n) return BsCand{pass ? OP_OR : OP_AND, st[i] + g / cn[j], st[j] + g % cn[j]};
      g -= n;
    }
  }
  return r;
}

__global__ void k_bs_base(BsDev D, unsigned long long nrows);
__global__ void k_bs_level(BsDev D, int c, unsigned long long cands);
__global__ void k_bs_mark(BsDev D, int c, unsigned long long cap, unsigned long long limit);
__global__ void k_bs_count(BsDev D, unsigned long long nwords);
__global__ void k_bs_offsets(BsDev D, unsigned chunks);
__global__ void k_bs_emit(BsDev D, unsigned long long nwords, unsigned long long out0);
__global__ void k_bs_vals(BsDev D, int c, unsigned long long out0);
__global__ void k_bs_bounds(BsDev D, const unsigned long long* rows_at, int n, unsigned long long* out);
__global__ void k_bs_leaves(const InstDev* I, const unsigned long long* rows, int n, int16_t* rpn, int* len);

// Set-up and maintenance kernels.
__global__ void k_fill(const __grid_constant__ BatchDev B);
__global__ void k_init(const __grid_constant__ BatchDev B);
__global__ void k_rehash(const Slot* old_tab, unsigned long long old_cap, Slot* new_tab,
                         unsigned long long new_mask, unsigned long long* fail);

}  // namespace vfb
