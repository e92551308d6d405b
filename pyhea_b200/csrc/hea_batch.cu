// hea_batch.cu -- the job engine's kernels (hea_batch.h says how they work).
#include "hea_batch.h"

namespace hea {

// Stable ascending order of order[0, count) by f2 (rank counting); block-wide,
// barriers inside.  scratch holds `count` ints.  Reads go through L2: the
// values were written by other CTAs of the same launch.
__device__ __forceinline__ void block_stable_sort(int32_t *order, const double *f2, int count, int32_t *scratch)
{
    for (int i = threadIdx.x; i < count; i += blockDim.x) scratch[i] = __ldcg(order + i);
    __syncthreads();
    for (int i = threadIdx.x; i < count; i += blockDim.x) {
        const double fi = __ldcg(f2 + __ldcg(scratch + i));
        int r = 0;
        for (int j = 0; j < count; ++j) {
            const double fj = __ldcg(f2 + __ldcg(scratch + j));
            r += (fj < fi) || (fj == fi && j < i);
        }
        order[r] = __ldcg(scratch + i);
    }
    __threadfence();
    __syncthreads();
}

__device__ __forceinline__ BatchJob &ring_slot(BatchJob *jobs, const BatchQueue &q, unsigned long long h)
{
    return jobs[q.base + h % q.cap];
}

// Append `n` fresh jobs of one kind for structure s to ring `level`
// (block-wide; thread 0 reserves the positions).
__device__ __forceinline__ void enqueue_jobs(BatchJob *jobs, BatchCtl *ctl, int level, int s, int kind, int iter,
                                             int n, unsigned long long *first_sh)
{
    if (threadIdx.x == 0) *first_sh = atomicAdd(&ctl->q[level].tail, (unsigned long long)n);
    __syncthreads();
    const unsigned long long first = *first_sh;
    const BatchQueue &q = ctl->q[level];
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
    const unsigned long long h = atomicAdd(&ctl->q[level].tail, 1ull);
    BatchJob &j = ring_slot(jobs, ctl->q[level], h);
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

// Thread 0: take the next reserved job of the highest level that has one.
// Returns its slot and expected sequence number, or -1 when no structure is
// active, the deadline has passed, or on error.
__device__ __forceinline__ long long claim_job(BatchCtl *ctl, unsigned long long deadline, int32_t *seq)
{
    const unsigned long long t0 = global_ns();
    for (;;) {
        if (*(volatile int32_t *)&ctl->active <= 0 || *(volatile int32_t *)&ctl->error) return -1;
        const unsigned long long now = global_ns();
        if (deadline && now >= deadline) return -1;
        for (int l = 0; l < kBatchLevels; ++l) {
            volatile BatchQueue *q = &ctl->q[l];
            unsigned long long h = q->head;
            while (h < q->tail) {
                const unsigned long long old = atomicCAS(&ctl->q[l].head, h, h + 1);
                if (old == h) {
                    *seq = (int32_t)(uint32_t)(h + 1);
                    return (long long)(q->base + h % q->cap);
                }
                h = old;
            }
        }
        const unsigned long long prog = *(volatile unsigned long long *)&ctl->progress_ns;
        const unsigned long long since = prog > t0 ? prog : t0;  // another SM's clock read may be ahead of ours
        if (now > since && now - since > ctl->wait_limit_ns) {
            atomicExch(&ctl->error, 1);
            return -1;
        }
        __nanosleep(256);
    }
}

// Phase-0 jobs of structures list[0, gridDim.x) (all structures when list is
// NULL); one CTA per structure.
__global__ void batch_seed_kernel(const BatchStruct *structs, const int32_t *list, BatchState *states, BatchJob *jobs,
                                  BatchCtl *ctl)
{
    __shared__ unsigned long long first;
    const int s = list ? list[blockIdx.x] : (int)blockIdx.x;
    const BatchStruct &d = structs[s];
    if (threadIdx.x == 0) {
        BatchState &st = states[s];
        st.remaining = d.I > 0 ? 2 * d.P : d.P;
        st.phase = 0;
        st.done = 0;
        st.tally[0] = st.tally[1] = st.tally[2] = 0;
        __threadfence();
        atomicAdd(&ctl->active, 1);
    }
    for (int i = threadIdx.x; i < 2 * d.P; i += blockDim.x) d.order[i] = i;
    __syncthreads();
    enqueue_jobs(jobs, ctl, d.level, s, kJobGen0, 0, d.P, &first);
    if (d.I > 0) enqueue_jobs(jobs, ctl, d.level, s, kJobGenMc, 0, d.P, &first);
}

struct JobEnd {
    int32_t yielded, round, miss;
};

// One job of a structure with species count T and layout L.  Shared memory:
// [occ (occ_stride + 16), unless hbm] | search_smem_tail(T, S, nwarps) (delta
// table, swap records, two count buffers).
// The rounds of a job's local search in a call of their own: values the job
// needs only before and after the search stay out of the loop's registers.
// One recount instance for the layouts that share it.
template <int T, int S, RecountForm kNeighbors>
__device__ __noinline__ void batch_recount(const SearchConst &c, const int4 *nbor, const uint8_t *occ, int32_t *cnt,
                                           uint64_t *hist)
{
    block_recount<T, S, kNeighbors>(c, nbor, occ, cnt, hist);
}

template <int T, class L>
__device__ __noinline__ McTally batch_search(const SearchConst &c, const BatchStruct &d, uint8_t *occ, int32_t *cnt2,
                                             const DeltaTab<T, L::S> tab, void *rec, uint32_t stream, double cur,
                                             const McResume rs, uint64_t *hist)
{
    return mc_rounds<T, L, false, true>(c, d.nbor, occ, cnt2, tab, rec, stream, cur, d.Q, d.D, d.max_rounds,
                                 McTrace{nullptr, nullptr, 0}, rs, hist, d.nbmask);
}

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
    const int slot = __ldcg(d.order + (job.kind == kJobGenMc ? P + pos : pos));
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
// launch's deadline has passed.  Dynamic shared memory: occupancy of the
// largest shared-memory structure + 16 + per-warp counts + swap records; the
// job's constants (1.9 KB) are copied to static shared memory.
__global__ void __launch_bounds__(HEA_BATCH_THREADS, HEA_BATCH_MIN_BLOCKS)
    batch_kernel(const BatchStruct *__restrict__ structs, BatchState *states, BatchJob *jobs, BatchCtl *ctl,
                 unsigned long long *finish_ns)
{
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ BatchJob job;
    __shared__ int stop, last, phase;
    __shared__ unsigned long long first;
    __shared__ __align__(16) SearchConst c;  // this job's constants: fitness tables read from shared memory
    const unsigned long long deadline = ctl->deadline_ns;  // set before the launch
    for (;;) {
        if (threadIdx.x == 0) {
            stop = 0;
            int32_t seq = 0;
            const long long h = claim_job(ctl, deadline, &seq);
            if (h < 0) {
                stop = 1;
            } else {
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
        __syncthreads();
        if (stop) break;
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
        if (threadIdx.x == 0) {
            if (e.yielded) {
                enqueue_resume(jobs, ctl, d.level, job, e.round, e.miss);
                last = 0;
            } else {
                last = atomicSub(&states[job.structure].remaining, 1) == 1;
                atomicMax(&ctl->progress_ns, global_ns());
                if (last) {
                    __threadfence();
                    phase = __ldcg(&states[job.structure].phase);
                }
            }
        }
        __syncthreads();
        if (!last) continue;
        // phase transition of this structure
        const int s = job.structure, P = d.P, I = d.I, k = phase;
        bool finished = (k == 0 && I == 0);  // generation 0 only: the reference returns it unsorted
        if (!finished) {
            if (k > 0) block_stable_sort(d.order, d.f2, P, d.scratch);  // survivors after their search
            if (k == I)
                finished = true;
            else if (k > 0 && d.tol2 >= 0.0 && __ldcg(d.f2 + __ldcg(d.order)) <= d.tol2)
                finished = true;  // tolerance reached
            else
                block_stable_sort(d.order, d.f2, 2 * P, d.scratch);  // merge of iteration k
        }
        if (finished) {
            if (threadIdx.x == 0) {
                finish_ns[s] = global_ns() - ctl->start_ns;
                states[s].done = 1;
                __threadfence();
                atomicAdd(&ctl->stats[3], 1ull);
                atomicSub(&ctl->active, 1);
            }
            __syncthreads();
            continue;
        }
        if (threadIdx.x == 0) {
            states[s].phase = k + 1;
            states[s].remaining = (k + 1 < I) ? 2 * P : P;
            __threadfence();
        }
        __syncthreads();
        enqueue_jobs(jobs, ctl, d.level, s, kJobMc2, k, P, &first);
        if (k + 1 < I) enqueue_jobs(jobs, ctl, d.level, s, kJobGenMc, k + 1, P, &first);
    }
}

BatchFn batch_kernel_fn() { return batch_kernel; }
BatchSeedFn batch_seed_kernel_fn() { return batch_seed_kernel; }

}  // namespace hea
