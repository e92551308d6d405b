// hea_batch.cu -- the job engine's kernels (hea_batch.h says how they work).
#include "hea_batch.h"

namespace hea {

// Stable ascending order by f2 (rank counting) of the slots a[0, na) followed by
// b[0, nb), both rewritten in rank order; block-wide, barriers inside.  scratch
// holds na + nb ints.  Reads go through L2: the values were written by other
// CTAs of the same launch.
__device__ __forceinline__ void block_stable_sort(int32_t *a, int na, int32_t *b, int nb, const double *f2,
                                                  int32_t *scratch)
{
    const int count = na + nb;
    for (int i = threadIdx.x; i < count; i += blockDim.x) scratch[i] = __ldcg(i < na ? a + i : b + (i - na));
    __syncthreads();
    for (int i = threadIdx.x; i < count; i += blockDim.x) {
        const double fi = __ldcg(f2 + __ldcg(scratch + i));
        int r = 0;
        for (int j = 0; j < count; ++j) {
            const double fj = __ldcg(f2 + __ldcg(scratch + j));
            r += (fj < fi) || (fj == fi && j < i);
        }
        *(r < na ? a + r : b + (r - na)) = __ldcg(scratch + i);
    }
    __threadfence();
    __syncthreads();
}

__device__ __forceinline__ int job_ring(int level, int kind) { return 2 * level + (kind == kJobGenMc); }

__device__ __forceinline__ BatchJob &ring_slot(BatchJob *jobs, const BatchQueue &q, unsigned long long h)
{
    return jobs[q.base + h % q.cap];
}

// Append `n` fresh jobs of one kind for structure s to its ring of `level`
// (block-wide; thread 0 reserves the positions).
__device__ __forceinline__ void enqueue_jobs(BatchJob *jobs, BatchCtl *ctl, int level, int s, int kind, int iter,
                                             int n, unsigned long long *first_sh)
{
    BatchQueue &q = ctl->q[job_ring(level, kind)];
    if (threadIdx.x == 0) *first_sh = atomicAdd(&q.tail, (unsigned long long)n);
    __syncwarp();
    __syncthreads();
    const unsigned long long first = *first_sh;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const unsigned long long h = first + i;
        BatchJob &j = ring_slot(jobs, q, h);
        j.structure = s;
        j.kind = kind;
        j.index = i;
        j.iter = iter;
        j.resume = 0;
        j.round0 = 0;
        j.miss0 = 0;
        __threadfence();
        atomicExch(&j.seq, (int32_t)(uint32_t)(h + 1));
    }
    __syncthreads();
}

// Thread 0: the continuation of a stopped local search.
__device__ __forceinline__ void enqueue_resume(BatchJob *jobs, BatchCtl *ctl, int level, const BatchJob &job,
                                               int64_t round0, int miss0)
{
    BatchQueue &q = ctl->q[job_ring(level, job.kind)];
    const unsigned long long h = atomicAdd(&q.tail, 1ull);
    BatchJob &j = ring_slot(jobs, q, h);
    j.structure = job.structure;
    j.kind = job.kind;
    j.index = job.index;
    j.iter = job.iter;
    j.resume = 1;
    j.round0 = (int32_t)round0;
    j.miss0 = miss0;
    __threadfence();
    atomicExch(&j.seq, (int32_t)(uint32_t)(h + 1));
}

// The block's first warp, converged: take the next reserved job of the first
// ring that has one; lane l looks at ring l, so a look costs one round trip to
// L2 however far down the work is.  Returns its slot and expected sequence
// number (every lane), or -1 when no structure is active, the deadline has
// passed, or on error.
__device__ __forceinline__ long long claim_job(BatchCtl *ctl, unsigned long long deadline, int32_t *seq)
{
    const int lane = threadIdx.x & 31;
    const unsigned long long t0 = global_ns();
    volatile BatchQueue *q = &ctl->q[lane];
    for (;;) {
        // head before tail: the pair never shows a job that was not reserved
        const unsigned long long head = q->head, tail = q->tail;
        int out = 0;  // lane 0: why to stop
        unsigned long long now = 0;
        if (lane == 0) {
            now = global_ns();
            if (*(volatile int32_t *)&ctl->active <= 0 || *(volatile int32_t *)&ctl->error || (deadline && now >= deadline))
                out = 1;
        }
        if (__shfl_sync(0xFFFFFFFFu, out, 0)) return -1;
        const uint32_t ready = __ballot_sync(0xFFFFFFFFu, head < tail);
        if (ready) {
            const int ring = __ffs(ready) - 1;
            unsigned long long mine = head;
            int won = 0;
            if (lane == ring)
                while (!won && mine < tail) {
                    const unsigned long long old = atomicCAS(&ctl->q[ring].head, mine, mine + 1);
                    won = old == mine;
                    if (!won) mine = old;  // another CTA took it: try the next
                }
            __syncwarp();
            if (__shfl_sync(0xFFFFFFFFu, won, ring)) {
                const unsigned long long h = __shfl_sync(0xFFFFFFFFu, mine, ring);
                *seq = (int32_t)(uint32_t)(h + 1);
                return (long long)(ctl->q[ring].base + h % ctl->q[ring].cap);
            }
            continue;  // others took them all
        }
        if (lane == 0) {
            const unsigned long long prog = *(volatile unsigned long long *)&ctl->progress_ns;
            const unsigned long long since = prog > t0 ? prog : t0;  // another SM's clock read may be ahead of ours
            if (now > since && now - since > ctl->wait_limit_ns) {
                atomicExch(&ctl->error, 1);
                out = 1;
            }
        }
        if (__shfl_sync(0xFFFFFFFFu, out, 0)) return -1;
        __nanosleep(256);
    }
}

// First jobs of structures list[0, gridDim.x) (all structures when list is
// NULL); one CTA per structure.
__global__ void batch_seed_kernel(const BatchStruct *structs, const int32_t *list, BatchState *states, BatchJob *jobs,
                                  BatchCtl *ctl)
{
    __shared__ unsigned long long first;
    const int s = list ? list[blockIdx.x] : (int)blockIdx.x;
    const BatchStruct &d = structs[s];
    const int ahead = min(d.ahead, d.I);
    if (threadIdx.x == 0) {
        BatchState &st = states[s];
        st.survivors = d.P;
        for (int r = 0; r < kBatchAhead; ++r) {
            st.left[r] = r < ahead ? d.P : 0;
            st.join[r] = 0;
        }
        st.iter = -1;
        st.phase = 0;
        st.done = 0;
        st.tally[0] = st.tally[1] = st.tally[2] = 0;
        __threadfence();
        atomicAdd(&ctl->active, 1);
    }
    for (int i = threadIdx.x; i < (d.ahead + 1) * d.P; i += blockDim.x) d.order[i] = i;
    __syncthreads();
    enqueue_jobs(jobs, ctl, d.level, s, kJobGen0, 0, d.P, &first);
    for (int it = 0; it < ahead; ++it) enqueue_jobs(jobs, ctl, d.level, s, kJobGenMc, it, d.P, &first);
}

struct JobEnd {
    int32_t yielded, round, miss;
};

// One recount instance for the layouts that share it.
template <int T, int S, RecountForm kNeighbors>
__device__ __noinline__ void batch_recount(const SearchConst &c, const int4 *nbor, const uint8_t *occ, int32_t *cnt,
                                           uint64_t *hist)
{
    block_recount<T, S, kNeighbors>(c, nbor, occ, cnt, hist);
}

// The rounds of a job's local search in a call of their own: values the job
// needs only before and after the search stay out of the loop's registers.
template <int T, class L>
__device__ __noinline__ McTally batch_search(const SearchConst &c, const BatchStruct &d, uint8_t *occ, int32_t *cnt2,
                                             const DeltaTab<T, L::S> tab, void *rec, uint32_t stream, double cur,
                                             const McResume rs, uint64_t *hist)
{
    return mc_rounds<T, L, true>(c, d.nbor, occ, cnt2, tab, rec, stream, cur, d.Q, d.D, d.max_rounds,
                                 McTrace{nullptr, nullptr, 0}, rs, hist, d.nbmask);
}

// One job of a structure with species count T and layout L.  Shared memory:
// [occ (occ_stride + 16), unless hbm] | search_smem_tail(T, S, nwarps) (delta
// table, swap records, two count buffers).
template <int T, class L>
__device__ __noinline__ JobEnd batch_job(const SearchConst &c, const BatchStruct &d, const BatchJob &job,
                                         uint8_t *smem, unsigned long long *stats, unsigned long long *tally,
                                         unsigned long long deadline)
{
    constexpr int S = L::S, NC = S * T * T, NCP = mc_ncount_pad(NC);
    const int nwarps = blockDim.x >> 5;
    const bool hbm = d.hbm != 0;
    const int P = d.P, n = c.num_sites;
    const int pos = job.index;
    const int slot = __ldcg(d.order + (job.kind == kJobGenMc ? P * (job.iter % d.ahead + 1) + pos : pos));
    uint8_t *gocc = d.occ + (size_t)slot * c.occ_stride;
    int32_t *gcnt = d.cnt + (size_t)slot * NC;
    uint64_t *hist = d.hist + (size_t)slot * c.num_sites * hist_words(T, S, L::kImplicit);
    uint8_t *occ = hbm ? gocc : smem;
    const DeltaTab<T, S> tab{reinterpret_cast<float *>(hbm ? smem : smem + c.occ_stride + 16)};
    uint8_t *rec = reinterpret_cast<uint8_t *>(tab.f + DeltaTab<T, S>::kFloats);  // [2][nwarps] records
    int32_t *cnt2 = reinterpret_cast<int32_t *>(rec + 2 * nwarps * record_bytes(T, S));

    double cur;
    if (job.kind == kJobMc2 || job.resume) {
        copy_occupancy<true>(c, gocc, occ);  // onto itself when hbm
        for (int x = threadIdx.x; x < NC; x += blockDim.x) cnt2[x] = __ldcg(gcnt + x);
        __syncthreads();
        if (threadIdx.x == 0) occ[n] = 0;  // sentinel
        cur = __ldcg(d.f2 + slot);  // a resumed search's running f2
    } else {
        const uint32_t generation = job.kind == kJobGen0 ? 0u : (uint32_t)(job.iter + 1);
        generate_occupancy<T>(c, (uint32_t)pos, generation, occ, (job.kind == kJobGen0 && !hbm) ? gocc : nullptr);
        if (threadIdx.x == 0) occ[n] = 0;
        __syncthreads();
        batch_recount<T, S, L::kImplicit ? kRecountLattice : kRecountTable>(c, d.nbor, occ, cnt2, hist);  // count buffer 0; ends with a barrier
        cur = fitness_of_counts<T, S>(c, cnt2);
        if (job.kind == kJobGen0) {
            for (int x = threadIdx.x; x < NC; x += blockDim.x) gcnt[x] = cnt2[x];
            if (threadIdx.x == 0) d.f2[slot] = cur;
            return JobEnd{0, 0, 0};
        }
    }
    search_setup<T, S>(c, cnt2, tab);
    const uint32_t call = job.kind == kJobMc2 ? (uint32_t)(2 * job.iter + 1) : (uint32_t)(2 * job.iter);
    const uint32_t stream = (call << 16) | (uint32_t)pos;
    const McResume rs{job.resume ? (int64_t)job.round0 : 0, job.resume ? job.miss0 : 0, deadline, d.tol2};
    // the draws read the species from the occupancy: measured on the mixed batch, the histograms'
    // species bits (draw_pair_hist) were slower for every structure size
    const McTally t = batch_search<T, L>(c, d, occ, cnt2, tab, rec, stream, cur, rs, hist);
    if (!hbm) copy_occupancy(c, occ, gocc);
    for (int x = threadIdx.x; x < NC; x += blockDim.x) gcnt[x] = cnt2[t.buf * NCP + x];
    add_tally(t, stats);
    add_tally(t, tally);
    if (threadIdx.x == 0) d.f2[slot] = t.f2;  // McTally::f2
    return JobEnd{t.yielded ? 1 : 0, (int32_t)t.round_end, t.miss};
}

template <int T>
__device__ __forceinline__ JobEnd batch_dispatch_t(const SearchConst &c, const BatchStruct &d, const BatchJob &job,
                                                   uint8_t *smem, unsigned long long *stats, unsigned long long *tally,
                                                   unsigned long long deadline)
{
    switch (d.layout) {
    case kLayBcc: return batch_job<T, Shells<2, 2, 3>>(c, d, job, smem, stats, tally, deadline);
    case kLayFccTrue: return batch_job<T, Shells<3, 2, 6>>(c, d, job, smem, stats, tally, deadline);
    case kLayRt1: return batch_job<T, RuntimeShells<1>>(c, d, job, smem, stats, tally, deadline);
    case kLayRt2: return batch_job<T, RuntimeShells<2>>(c, d, job, smem, stats, tally, deadline);
    case kLayImp1: return batch_job<T, ImplicitShells<1>>(c, d, job, smem, stats, tally, deadline);
    case kLayImp2: return batch_job<T, ImplicitShells<2>>(c, d, job, smem, stats, tally, deadline);
    case kLayImp3: return batch_job<T, ImplicitShells<3>>(c, d, job, smem, stats, tally, deadline);
    default: return batch_job<T, RuntimeShells<3>>(c, d, job, smem, stats, tally, deadline);
    }
}

// The persistent kernel: CTAs take jobs until no structure is active or the
// launch's deadline has passed.
//
// Barriers.  Every path through the loop body meets the same barriers in every
// warp: what decides a path (stop, last, merge, finished) is the same value in
// all threads, from a barrier or from shared memory behind one.  Shared values
// are written by thread 0 before the barrier that publishes them and not again
// until the CTA has met another one behind their last read: job, merge, behind
// (read behind the barrier on `last`; the next job's barriers follow), first
// (enqueue_jobs ends with one), c.  Block barriers are instructions of whole
// warps, so where thread 0 works alone (a wait for a producer, a transition's
// counts) its warp comes together first (__syncwarp): lanes that reached the
// barrier ahead of it would count their warp as arrived, and the other warps
// would go on with the job that stood there before.  That would explain what an
// earlier form without it, with a plain barrier and a shared stop flag, once
// did (other warps took the old job again); the form is not run any more, so it
// is an explanation and not a finding.
//
// Dynamic shared memory: what the largest job needs (batch_job: staged occupancy,
// delta table, swap records, count buffers); the job's constants (SearchConst,
// 2.1 KB) are copied to static shared memory.
__global__ void __launch_bounds__(HEA_BATCH_THREADS, HEA_BATCH_MIN_BLOCKS)
    batch_kernel(const BatchStruct *__restrict__ structs, BatchState *states, BatchJob *jobs, BatchCtl *ctl,
                 unsigned long long *finish_ns)
{
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ BatchJob job;
    __shared__ int merge, behind;
    __shared__ unsigned long long first;
    __shared__ __align__(16) SearchConst c;  // this job's constants: fitness tables read from shared memory
    const unsigned long long deadline = ctl->deadline_ns;  // set before the launch
    for (;;) {
        int32_t seq = 0;
        const long long h = threadIdx.x < 32 ? claim_job(ctl, deadline, &seq) : 0;
        int stop = h < 0;  // thread 0's counts
        if (threadIdx.x == 0) {
            if (h >= 0) {
                volatile int32_t *vs = &jobs[h].seq;
                const unsigned long long t0 = global_ns();
                while (*vs != seq) {  // the producer reserved this position and is filling it
                    if (*(volatile int32_t *)&ctl->error || global_ns() - t0 > ctl->wait_limit_ns) {
                        atomicCAS(&ctl->error, 0, 1);
                        stop = 1;
                        break;
                    }
                    __nanosleep(64);
                }
                if (!stop) {
                    __threadfence();
                    const BatchJob *src = &jobs[h];
                    job.structure = __ldcg(&src->structure);
                    job.kind = __ldcg(&src->kind);
                    job.index = __ldcg(&src->index);
                    job.iter = __ldcg(&src->iter);
                    job.resume = __ldcg(&src->resume);
                    job.round0 = __ldcg(&src->round0);
                    job.miss0 = __ldcg(&src->miss0);
                    __threadfence();
                    if (*vs != seq) {  // reused before it was read: the ring is too small
                        atomicCAS(&ctl->error, 0, 2);
                        stop = 1;
                    }
                }
            }
        }
        // Thread 0's answer travels in the barrier, which needs no shared flag.
        __syncwarp();
        if (__syncthreads_or(threadIdx.x == 0 && stop)) break;
        // this job's structure: read-only while it is active
        const BatchStruct &d = structs[job.structure];
        {  // 8-byte words: SearchConst holds doubles, so it is 8-byte aligned and sized
            const int2 *src = reinterpret_cast<const int2 *>(&d.c);
            int2 *dst = reinterpret_cast<int2 *>(&c);
            for (int x = threadIdx.x; x < (int)(sizeof(SearchConst) / 8); x += blockDim.x) dst[x] = __ldg(src + x);
        }
        __syncthreads();
        unsigned long long *tally = states[job.structure].tally;
        JobEnd e;
        switch (d.T) {
        case 2: e = batch_dispatch_t<2>(c, d, job, smem, ctl->stats, tally, deadline); break;
        case 3: e = batch_dispatch_t<3>(c, d, job, smem, ctl->stats, tally, deadline); break;
        case 4: e = batch_dispatch_t<4>(c, d, job, smem, ctl->stats, tally, deadline); break;
        case 5: e = batch_dispatch_t<5>(c, d, job, smem, ctl->stats, tally, deadline); break;
        default: e = batch_dispatch_t<6>(c, d, job, smem, ctl->stats, tally, deadline); break;
        }
        __threadfence();  // every writer orders its results before the completion count
        __syncthreads();
        // the last job of its kind runs the structure's transition; merge: the iteration to merge, or -1
        const int s = job.structure, P = d.P, I = d.I;
        BatchState &st = states[s];
        const bool population = job.kind == kJobGenMc;
        int last = 0;  // thread 0's counts
        if (threadIdx.x == 0) {
            merge = -1;
            if (e.yielded) {
                enqueue_resume(jobs, ctl, d.level, job, e.round, e.miss);
            } else {
                last = atomicSub(population ? &st.left[job.iter % d.ahead] : &st.survivors, 1) == 1;
                atomicMax(&ctl->progress_ns, global_ns());
                if (last) __threadfence();
                if (last && !population) behind = __ldcg(&st.iter) + 1;
                if (last && population) {
                    if (atomicAdd(&st.join[job.iter % d.ahead], 1) == 1) merge = job.iter;
                }
            }
        }
        __syncwarp();
        if (!__syncthreads_or(threadIdx.x == 0 && last)) continue;
        bool finished = false;
        if (!population) {
            // iterations the survivors have behind them, read once: another CTA may merge and count on
            // as soon as the token below is in
            const int k = behind;
            if (k > 0) block_stable_sort(d.order, P, nullptr, 0, d.f2, d.scratch);
            finished = k == I;  // with I = 0, generation 0 only: the reference returns it unsorted
            if (!finished && threadIdx.x == 0) {
                __threadfence();
                if (atomicAdd(&st.join[k % d.ahead], 1) == 1) merge = k;
            }
            if (finished && threadIdx.x == 0) st.phase = k;
            __syncwarp();
            __syncthreads();
        }
        const int it = merge;
        if (!finished && it < 0) continue;  // the other token comes later
        if (!finished) {
            __threadfence();
            if (it > 0 && d.tol2 >= 0.0 && __ldcg(d.f2 + __ldcg(d.order)) <= d.tol2) {
                finished = true;  // tolerance reached
                if (threadIdx.x == 0) st.phase = it;
                __syncwarp();
            } else {
                block_stable_sort(d.order, P, d.order + (size_t)P * (it % d.ahead + 1), P, d.f2, d.scratch);
            }
        }
        if (finished) {
            if (threadIdx.x == 0) {
                finish_ns[s] = global_ns() - ctl->start_ns;
                st.done = 1;
                __threadfence();
                atomicAdd(&ctl->stats[3], 1ull);
                atomicSub(&ctl->active, 1);
            }
            __syncwarp();
            __syncthreads();
            continue;
        }
        const bool more = it + d.ahead < I;  // another population into the slots the merge freed
        if (threadIdx.x == 0) {
            st.iter = it;
            st.survivors = P;
            st.join[it % d.ahead] = 0;
            if (more) st.left[it % d.ahead] = P;
            __threadfence();
        }
        __syncwarp();
        __syncthreads();
        enqueue_jobs(jobs, ctl, d.level, s, kJobMc2, it, P, &first);
        if (more) enqueue_jobs(jobs, ctl, d.level, s, kJobGenMc, it + d.ahead, P, &first);
    }
}

BatchFn batch_kernel_fn() { return batch_kernel; }
BatchSeedFn batch_seed_kernel_fn() { return batch_seed_kernel; }

}  // namespace hea
