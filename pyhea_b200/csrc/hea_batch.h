// hea_batch.h -- the job engine: many independent structures searched by one
// persistent kernel.  It serves both the batch API (hea_batch_*: a fixed set
// of structures in one graph-captured launch) and the serving loop
// (hea_server_*: structures admitted while others run, in time slices).
//
// Every structure runs the same search as the plain path (hea_search.cuh) with
// its own constants, tables, population pools and Philox key, so its result
// is bit-identical to searching it alone, whatever else shares the GPU.  Its
// work is a graph of jobs, P of each kind and iteration:
//
//   GEN0           generation 0: the first survivors
//   GENMC(i)       generation i + 1, then its local search (mc_call 2i): the new
//                  population of iteration i, in slots of ring i mod W
//   MC2(i)         local search of the survivors of iteration i's merge
//                  (mc_call 2i + 1)
//
// A new population depends on nothing but the seed, so W of them (`ahead`) are
// queued from the start; iteration i's merge waits for population i and for the
// survivors of iteration i - 1 (two tokens, BatchState::join), and frees
// population i's slots for population i + W.  So a structure's chain is one long
// search and I short ones, not I long ones, and its long searches fill the chip.
// The CTA that finishes the last job of a kind, or brings the second token, runs
// the transition itself -- stable sort of the survivors, then the merge
// (pyhea/cpp/accelerate.cpp:305-330, :693) -- and appends the jobs it frees.
// With a tolerance, a local search also ends once its f2 is at or below it, and
// the structure ends at the merge that finds the survivors' best f2 at or below
// it (the population it waited for is dropped); W is then 1, so that no more
// than that one is searched in vain.
//
// Jobs live in ring queues, two per priority level (survivors' jobs before new
// populations'), whose head and tail only grow; a CTA's first warp looks at all
// rings at once, takes the next reserved job of the first that has one and waits
// for the producer's sequence number in the slot.  A ring needs room for the
// unfinished jobs of its kind of every structure at its level (at most W P each).
//
// A launch ends when no structure is active or, for the time slices of the
// serving loop, at its deadline: CTAs stop taking jobs, and a local search
// that sees the deadline stops at the end of its round, saves its state
// (occupancy, counts, f2) to HBM and queues a continuation that resumes at
// the next round with the same rejection count -- the same proposals follow,
// so the result does not depend on where the slices fell.  Waits are bounded
// by wall time since the last finished job; on expiry the kernel sets an
// error flag and every CTA returns.
//
// Proposals are scored from the site histograms, so a search reads the occupancy
// only for its draws.  Where it lies is the host's choice (a batch stages every
// row in shared memory when all fit, else keeps all in HBM; a server by its
// hbm_sites, all in HBM unless set).  In HBM (`hbm`) a job copies the row onto itself (reads through L2,
// so no stale L1 line of another SM's writes is used; the copy rewrites every
// byte this CTA later reads) and searches it through L1.  Otherwise the row is
// staged in the launch's shared memory.
#pragma once
#include <cstdint>

#include "hea_search.cuh"

namespace hea {

enum BatchJobKind : int32_t { kJobGen0 = 0, kJobGenMc = 1, kJobMc2 = 2 };

struct BatchJob {
    int32_t structure, kind, index, iter;
    int32_t seq;     // low 32 bits of (ring position + 1), written after the other fields
    int32_t resume;  // 1: continue a stopped local search at round0 with miss0 rejections
    int32_t round0, miss0;
};
static_assert(sizeof(BatchJob) == 32, "BatchJob layout");

// Kernel instance of a structure: species count and shell layout.
enum BatchLayout : int32_t {
    kLayBcc = 0, kLayFccTrue = 1, kLayRt1 = 2, kLayRt2 = 3, kLayRt3 = 4, kLayImp1 = 5, kLayImp2 = 6, kLayImp3 = 7
};

struct BatchStruct {
    SearchConst c;
    const int4 *nbor;
    uint8_t *occ;
    int32_t *cnt;
    double *f2;
    int32_t *order;    // [P (W + 1)] slot ids: the survivors', then each new population's
    int32_t *scratch;  // [2P] sort scratch
    uint64_t *hist;    // [P (W + 1)][N] site histograms (SiteHist)
    const uint32_t *nbmask;
    int32_t P, Q, D, I;
    int64_t max_rounds;
    double tol2;  // tolerance on f2 (< 0: none): local searches and the structure end once reached
    int32_t T, layout, level, hbm;
    int32_t ahead, pad_;  // W: new populations in flight, 1..kBatchAhead
};

static_assert(sizeof(SearchConst) % 8 == 0 && alignof(SearchConst) >= 8, "SearchConst copied as 8-byte words");

constexpr int kBatchAhead = 4;

struct BatchState {
    int32_t survivors;          // survivors' jobs (GEN0 or MC2) not finished
    int32_t left[kBatchAhead];  // jobs of each new population not finished
    int32_t join[kBatchAhead];  // tokens of the merge of each: 2 once survivors and population are ready
    int32_t iter;               // iteration of the survivors' jobs (-1: GEN0)
    int32_t phase;              // at the end: the iterations run
    int32_t done;               // 1 once the structure's search ended
    unsigned long long tally[3];  // rounds, evals, accepts of this structure
};
static_assert(sizeof(BatchState) % 8 == 0, "BatchState copied whole");

constexpr int kBatchLevels = 16;

struct BatchQueue {
    unsigned long long head;  // jobs taken
    unsigned long long tail;  // jobs reserved by producers
    unsigned long long cap;   // ring slots
    unsigned long long base;  // first slot of this ring in the job array
};

constexpr int kBatchRings = 2 * kBatchLevels;  // ring 2 l: survivors' jobs of level l; 2 l + 1: new populations'
static_assert(kBatchRings == 32, "one lane per ring (claim_job)");

struct BatchCtl {
    BatchQueue q[kBatchRings];
    unsigned long long stats[4];  // rounds, evals, accepts, finished structures
    int32_t error;                // 1: a wait ran out of time, 2: a ring slot was overwritten
    int32_t active;               // structures seeded and not finished
    unsigned long long wait_limit_ns;
    unsigned long long start_ns;     // device time origin of finish times
    unsigned long long deadline_ns;  // device time after which no job starts (0: none)
    unsigned long long progress_ns;  // device time of the last finished job
};

#ifndef HEA_BATCH_THREADS
#define HEA_BATCH_THREADS 256
#endif
#ifndef HEA_BATCH_MIN_BLOCKS
#define HEA_BATCH_MIN_BLOCKS 3  // resident CTAs per SM the register budget aims for (measured: 3 > 2, 4)
#endif

// The kernels, compiled in a unit of their own (hea_batch.cu).
using BatchFn = void (*)(const BatchStruct *structs, BatchState *states, BatchJob *jobs, BatchCtl *ctl,
                         unsigned long long *finish_ns);
using BatchSeedFn = void (*)(const BatchStruct *structs, const int32_t *list, BatchState *states, BatchJob *jobs,
                             BatchCtl *ctl);
BatchFn batch_kernel_fn();
BatchSeedFn batch_seed_kernel_fn();

}  // namespace hea
