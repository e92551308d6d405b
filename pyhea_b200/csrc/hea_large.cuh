// hea_large.cuh -- the search for structures whose occupancy does not fit in
// shared memory (up to millions of sites).
//
// Same contract as hea_search.cuh (Philox streams, counts, fitness order,
// ties), so results are bit-identical to the shared-memory path; only where
// the occupancy lives and how many SMs work on one solution change:
//   * the occupancy row stays in HBM as species bytes; the local search does
//     not read or write it: its draws take the species from the site
//     histograms' species bits, which the accepts
//     keep current, and at its end each CTA writes its share of the row back
//     from those bits;
//   * one thread-block cluster per solution: the round's tasks are split over
//     the cluster's CTAs; each CTA reduces its warps' records, publishes its
//     best in shared memory, and after one cluster barrier every warp reads the
//     CL records through distributed shared memory and applies the same winner;
//   * generation and recount are grid-wide over sites (many CTAs per solution);
//     the recount also writes the site histograms the search scores from
//     (hist, see score_delta), which rank 0 of the cluster updates after every
//     accepted swap, followed by a cluster barrier that only rank 0 arrives at
//     with release semantics (the other CTAs have nothing to publish).
#pragma once
#include <cooperative_groups.h>

#include "hea_search.cuh"

namespace hea {

namespace cg = cooperative_groups;

// Random occupancy of population positions [0, count) of `generation` into
// slot rows order[pos], as species bytes.  grid = (chunks, count).
template <int T>
__global__ void __launch_bounds__(256) large_generate_kernel(const SearchConst c, uint8_t *occ, const int32_t *order,
                                                             uint32_t generation)
{
    const uint32_t pos = blockIdx.y;
    uint8_t *row = occ + (size_t)order[pos] * c.occ_stride;
    uint32_t rk[kFeistelRounds];
    const u32x4 w0 = philox4x32_10(u32x4{pos, generation, 0u, kInitStream}, c.key0, c.key1);
    const u32x4 w1 = philox4x32_10(u32x4{pos, generation, 1u, kInitStream}, c.key0, c.key1);
    rk[0] = w0.x; rk[1] = w0.y; rk[2] = w0.z; rk[3] = w0.w; rk[4] = w1.x; rk[5] = w1.y;
    const int n = c.num_sites;
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < n; s += gridDim.x * blockDim.x) {
        uint32_t y = feistel((uint32_t)s, c.feistel_h, rk);
        while (y >= (uint32_t)n) y = feistel(y, c.feistel_h, rk);
        int t = 0;
#pragma unroll
        for (int i = 1; i < T; ++i) t += (int)(y >= (uint32_t)c.prefix[i]);
        row[s] = (uint8_t)t;
    }
}

// Pair counts of slot rows order[pos] (species bytes), accumulated into
// cnt[order[pos]] (zeroed by the caller), and, with `hist`, the site
// histograms of those rows (hist + slot * N; see block_recount).  grid =
// (chunks, count); each CTA counts a range of sites into shared bins and adds
// them once.
template <int T, int S>
__global__ void __launch_bounds__(256) large_recount_kernel(const SearchConst c, const int4 *__restrict__ nbor,
                                                            const uint8_t *occ, const int32_t *order, int32_t *cnt,
                                                            uint64_t *hist)
{
    __shared__ int32_t bins[S * T * T];
    const int slot = order[blockIdx.y];
    const uint8_t *row = occ + (size_t)slot * c.occ_stride;
    for (int x = threadIdx.x; x < S * T * T; x += blockDim.x) bins[x] = 0;
    __syncthreads();
    const int n = c.num_sites;
    uint64_t *hs = hist ? hist + (size_t)slot * n * hist_words(T, S, c.lat.L > 0) : nullptr;
    // one site with its shell histograms h (5-bit fields)
    const auto site = [&](int s, const uint32_t (&h)[S], auto form) {
        using H = SiteHist<T, S, decltype(form)::value>;
        const int a = row[s];
#pragma unroll
        for (int k = 0; k < S; ++k) {
#pragma unroll
            for (int t = 0; t < T; ++t) {
                const int v = (int)((h[k] >> (5 * t)) & 31u);
                if (v) atomicAdd(&bins[(k * T + a) * T + t], v);
            }
        }
        if (hs) {
            const HistEntry<H::W> e = pack_hist<H, T, S, 5>(c, h, a);
#pragma unroll
            for (int x = 0; x < H::W; ++x) hs[(size_t)s * H::W + x] = e.w[x];
        }
    };
    const int first = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
    if (c.lat.L) {  // implicit neighbours (no sentinel padding: pad[k] == 0)
        lattice_sites<S, uint32_t>(c.lat, first, stride, [row](int n) { return 1u << (5 * row[n]); },
                                   [&site](int s, const uint32_t (&h)[S]) { site(s, h, std::true_type{}); });
    } else {
        for (int s = first; s < n; s += stride) {
            uint32_t h[S];
#pragma unroll
            for (int k = 0; k < S; ++k) {
                h[k] = 0;
                const int4 *seg = nbor + (size_t)s * c.row4 + c.off4[k];
                for (int ch = 0; ch < c.chunks[k]; ++ch) {
                    const int4 x = __ldg(seg + ch);
                    h[k] += (1u << (5 * row[x.x])) + (1u << (5 * row[x.y])) + (1u << (5 * row[x.z])) +
                            (1u << (5 * row[x.w]));
                }
            }
            site(s, h, std::false_type{});
        }
    }
    __syncthreads();
    int32_t *g = cnt + (size_t)slot * S * T * T;
    for (int x = threadIdx.x; x < S * T * T; x += blockDim.x) {
        int v = bins[x];
        if (blockIdx.x == 0 && x % T == 0) {  // sentinel entries land in field 0: pad_k per site of species i
            const int k = x / (T * T), i = (x / T) % T;
            v -= c.pad[k] * (c.prefix[i + 1] - c.prefix[i]);
        }
        if (v) atomicAdd(&g[x], v);
    }
}

// f2 of slots order[0, count) from their counts.
template <int T, int S>
__global__ void large_fitness_kernel(const SearchConst c, const int32_t *order, int count, const int32_t *cnt,
                                     double *f2)
{
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= count) return;
    const int slot = order[p];
    f2[slot] = fitness_of_counts<T, S>(c, cnt + (size_t)slot * S * T * T);
}

// The local search with the occupancy in HBM, one cluster per solution.
// Shared memory: search_smem_tail(T, S, nwarps) + 2 * record_bytes(T, S):
// delta table, the warps' records [2][nwarps], this CTA's best record [2]
// (read by the cluster), and two count buffers.  Every CTA keeps its own copy of
// the table and counts and applies each accepted swap to them itself.
template <int T, class L>
__global__ void __launch_bounds__(512, 2) mc_large_kernel(const __grid_constant__ SearchConst c, const McArgs g)
{
    constexpr int S = L::S, NC = S * T * T, NCP = mc_ncount_pad(NC);
    constexpr int W = SiteHist<T, S, L::kImplicit>::W;
    using H = SiteHist<T, S, L::kImplicit>;
    using Record = SwapRecord<W>;
    extern __shared__ __align__(16) uint8_t smem[];
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = (int)cluster.block_rank(), csize = (int)cluster.num_blocks();
    const int sol = blockIdx.x / csize;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
    const DeltaTab<T, S> tab{reinterpret_cast<float *>(smem)};
    Record *rec = reinterpret_cast<Record *>(tab.f + DeltaTab<T, S>::kFloats);  // [2][nwarps]
    Record *cta_rec = rec + 2 * nwarps;                                   // [2]: this CTA's best
    int32_t *cnt2 = reinterpret_cast<int32_t *>(cta_rec + 2);             // [2][NCP]

    const int slot = g.order[sol];
    const uint32_t stream = (g.mc_call << 16) | (uint32_t)sol;
    uint8_t *row = g.occ + (size_t)slot * c.occ_stride;
    uint64_t *hist = g.hist + (size_t)slot * c.num_sites * W;
    int32_t *gcnt = g.cnt + (size_t)slot * NC;
    const int n = c.num_sites;
    // this CTA's share of the row and of the tasks
    const int part = (n + csize - 1) / csize, row_lo = rank * part, row_hi = min(n, row_lo + part);
    const int qpart = (g.tasks + csize - 1) / csize, qlo = rank * qpart, qhi = min(g.tasks, qlo + qpart);

    for (int x = tid; x < NC; x += blockDim.x) cnt2[x] = gcnt[x];
    __syncthreads();
    search_setup<T, S>(c, cnt2, tab);
    cluster.sync();

    double cur = g.f2[slot];
    int miss = 0, buf = 0;
    int64_t round = 0, accepts = 0;
    uint32_t undrawn = 0;  // this thread's tasks that found no pair
    while (miss < g.depth && round < g.max_rounds) {
        Record *rr = rec + (round & 1) * nwarps;
        Record &mine = rr[warp];
        if (lane == 0) mine.lo = mine.hi = kEmpty;
        __syncwarp();
        const int32_t *cold = cnt2 + buf * NCP;
        for (int q0 = qlo + warp * 32; q0 < qhi; q0 += blockDim.x) {
            const int q = q0 + lane;
            uint32_t s1 = 0, s2 = 0;
            Record r;
            r.p = r.q = HistEntry<W>{};
            // the species come from the histograms' top bits: one L2 round trip per attempt
            const bool ok = q < qhi && draw_pair_hist<H>(c, stream, (uint32_t)round, (uint32_t)q, hist, s1, s2, r.p, r.q);
            __syncwarp();
            undrawn += q < qhi && !ok;
            const int a = hist_species<H>(r.p), b = hist_species<H>(r.q);
            r.ab = a | (b << 8);
            float B;
            const float D = score_delta<T, L>(c, g.nbor, g.nbmask, tab, r.p, r.q, s1, s2, a, b, B);
            screen_interval(c, tab, ok, D, B, r.lo, r.hi);
            r.task = q;
            r.s1 = s1;
            r.s2 = s2;
            r.stop = 0;
            r.pad_ = 0;
            keep_best<T, L>(c, cold, mine, r, q0 != qlo + warp * 32);
        }
        __syncthreads();
        // this CTA's best record, published for the cluster
        if (warp == 0) {
            const int xw = best_record<T, L>(c, cold, lane < nwarps ? rr[lane].lo : kNoSwap,
                                             lane < nwarps ? rr[lane].hi : kNoSwap, nwarps,
                                             [rr](int i) -> const Record & { return rr[i]; });
            if (lane == 0) {
                if (xw >= 0)
                    cta_rec[round & 1] = rr[xw];
                else
                    cta_rec[round & 1].lo = cta_rec[round & 1].hi = kNoSwap;
            }
        }
        __syncwarp();
        cluster.sync();
        // every warp reduces the cluster's records
        float lo = kNoSwap, hi = kNoSwap;
        if (lane < csize) {
            const Record *remote = cluster.map_shared_rank(&cta_rec[round & 1], lane);
            lo = remote->lo;
            hi = remote->hi;
        }
        const int xr = best_record<T, L>(c, cold, lo, hi, csize, [&cluster, cta_rec, round](int i) {
            return *cluster.map_shared_rank(&cta_rec[round & 1], i);
        });
        if (xr >= 0) {
            const Record w = *cluster.map_shared_rank(&cta_rec[round & 1], xr);
            const int a = w.ab & 0xFF, b = w.ab >> 8;
            int32_t *cnew = cnt2 + (buf ^ 1) * NCP;
            accept_counts<T, L>(tab, w, a, b, cold, cnew);
            if (rank == 0)
                update_hist<T, L, true>(c, g.nbor, hist, w.s1, w.s2, a, b, block_rotation(32 * DeltaTab<T, S>::kWarps));
            // the cluster's next proposals read the histograms and species bits rank 0 updated: rank 0
            // arrives with release semantics, the others (whose accept work stays in their own shared
            // memory, ordered by the block barrier) relaxed, every thread waits with acquire semantics.  Measured: 4 % per round.
            __syncwarp();
            __syncthreads();  // this CTA's warps read the new counts and table
            if (rank == 0)
                __cluster_barrier_arrive();
            else
                __cluster_barrier_arrive_relaxed();
            __cluster_barrier_wait();
            if (g.trace && rank == 0 && warp == 0) cur = __dadd_rn(cur, exact_delta<T, L>(c, cold, a, b, w.p, w.q));
            buf ^= 1;
            if (g.trace && rank == 0 && warp == 0 && accepts < g.trace_cap) {
                if (lane == 0) {
                    AcceptRecord r;
                    r.round = (uint32_t)round;
                    r.task = (uint32_t)w.task;
                    r.s1 = w.s1;
                    r.s2 = w.s2;
                    r.f2 = cur;
                    g.trace[(size_t)sol * g.trace_cap + accepts] = r;
                }
                if (g.trace_counts) {
                    int32_t *dst = g.trace_counts + ((size_t)sol * g.trace_cap + accepts) * NC;
                    for (int x = lane; x < NC; x += 32) dst[x] = cnew[x];
                }
            }
            miss = 0;
            ++accepts;
        } else {
            ++miss;
        }
        ++round;
    }
    cluster.sync();  // rank 0's last species bits are visible
    for (int s = row_lo + tid; s < row_hi; s += blockDim.x) {
        HistEntry<W> e, same;
        load_hist_pair<W>(c, hist, (uint32_t)s, (uint32_t)s, e, same);
        row[s] = (uint8_t)hist_species<H>(e);
    }
    if (rank == 0)
        for (int x = tid; x < NC; x += blockDim.x) gcnt[x] = cnt2[buf * NCP + x];
    const int share = max(0, qhi - qlo);  // this CTA's tasks
    const int64_t scored = (int64_t)(tid < share ? (share - 1 - tid) / (int)blockDim.x + 1 : 0) * round;
    unsigned long long ev = (unsigned long long)(scored - undrawn);
#pragma unroll
    for (int o = 16; o; o >>= 1) ev += __shfl_xor_sync(0xFFFFFFFFu, ev, o);
    if (lane == 0 && ev) atomicAdd(&g.stats[1], ev);
    if (rank == 0 && tid == 0) {
        g.f2[slot] = fitness_of_counts<T, S>(c, cnt2 + buf * NCP);
        atomicAdd(&g.stats[0], (unsigned long long)round);
        atomicAdd(&g.stats[2], (unsigned long long)accepts);
        if (g.trace_len) g.trace_len[sol] = accepts;
        if (g.rounds_out) g.rounds_out[sol] = round;
    }
    cluster.sync();  // keep every CTA's shared memory alive until all remote reads are done
}

}  // namespace hea
