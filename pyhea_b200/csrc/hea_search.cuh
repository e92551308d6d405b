// hea_search.cuh -- the swap-search kernels (sm_100a), templated on the number
// of species T and on the shell layout of the neighbour table.
//
// Layout in HBM (one structure):
//   nbor   int32 [N][row] with every shell segment padded to a multiple of 4
//          entries by the sentinel site N, so each segment is read as int4
//   occ    uint8 [slots][occ_stride]   species per site, one row per slot
//   cnt    int32 [slots][S][T][T]      pair counts that travel with their slot
//   f2     double [slots]              squared weighted SRO error
//   order  int32 [P (W + 1)]           slot ids: survivors, then each of W new populations
// In shared memory a slot's occupancy has the sentinel byte 0 at index N.
#pragma once
#include <cstdint>
#include <type_traits>
#include <utility>

#include "hea_device.cuh"

namespace hea {

// Implicit neighbour ids of a perfect FCC/BCC cube (the structure keeps no
// neighbour table in memory).  Site s = nb (cx L^2 + cy L + cz) + b is basis
// site b of cell (cx, cy, cz).  Its neighbours (shells concatenated) lie in
// cells (cx + dx, cy + dy, cz + dz), d in {-1, 0, 1}, periodic in every axis,
// at basis b' -- both fixed by the lattice's shell vectors.  Shell generators
// in half lattice units: FCC (1,1,0) 12, (2,0,0) 6, then (2,2,0) 12 (reference
// set) or (2,1,1) 24 (true third shell); BCC (1,1,1) 8, (2,0,0) 6, (2,2,0) 12.
// The sets equal the table of pyhea/lattice/lattice.py:196-323; entries of a
// shell come in another order, which no count or histogram sees.
struct LatticeConst {
    int32_t L;                   // cube edge in cells; 0: the structure has a neighbour table
    int32_t nb;                  // basis sites per cell (4 FCC, 2 BCC)
    int32_t zsize[3], zoff[3];   // shell sizes and offsets in the concatenated neighbour list
    uint32_t mul_L, mul_LL;      // floor(2^32 / L) and floor(2^32 / L^2) (lattice_cell)
    int32_t kind;                // kLatFccRef, kLatFccTrue3 or kLatBcc
    int32_t pad_;
};
static_assert(sizeof(LatticeConst) % 8 == 0, "LatticeConst keeps SearchConst 8-byte sized");

struct SearchConst {
    double E[kMaxShells * kMaxTypes * kMaxTypes];  // 1 - target, [S][T][T] compact
    double R[kMaxShells * kMaxTypes * kMaxTypes];  // N / (Z_k n_i n_j), [S][T][T] compact
    double w[kMaxShells];
    int32_t off4[kMaxShells];     // shell segment start in a row, int4 units
    int32_t chunks[kMaxShells];   // shell segment length, int4 units
    int32_t pad[kMaxShells];      // sentinel entries in the segment
    int32_t prefix[kMaxTypes + 1];  // species prefix sums
    int32_t num_sites, row4, occ_stride, num_types, num_shells, feistel_h;
    uint32_t key0, key1;
    uint32_t draw16;    // 1: 16-bit draws, four attempts per Philox call (use_draw16)
    uint32_t reject;    // draws whose product has a lower remainder are rejected: 2^32 mod N, or (2^16 mod N) << 16
    uint32_t hist_stream;  // 1: site histograms read with streaming (evict-first) loads (load_hist_pair)
    float screen_floor;    // 0; 3e38 when FP32's range does not hold the structure: every D is then exact
    double screen_scale;   // power of two that brings the largest Q to about 1 in the FP32 table
    float screen_sw[kMaxShells + 1];           // sqrt(w * screen_scale), rounded up
    float kappa[kMaxTypes * kMaxTypes];        // max(1, n_t / n_i) at [i][t], rounded up
    LatticeConst lat;   // lat.L > 0: neighbours from lattice arithmetic (nbor unused)
};

enum : int { kLatFccRef = 0, kLatFccTrue3 = 1, kLatBcc = 2 };

__host__ __device__ constexpr int lat_nb(int kind) { return kind == kLatBcc ? 2 : 4; }
__host__ __device__ constexpr int lat_basis(int kind, int b, int d)
{
    // half-unit basis offsets: FCC {0,0,0} {1,1,0} {1,0,1} {0,1,1}; BCC {0,0,0} {1,1,1}
    return kind == kLatBcc ? b : (b == 0 ? 0 : (d == 0 ? (b != 3) : d == 1 ? (b != 2) : (b != 1)));
}
__host__ __device__ constexpr int lat_gen(int kind, int k, int d)
{
    return k == 0 ? (kind == kLatBcc ? 1 : (d < 2 ? 1 : 0))
         : k == 1 ? (d == 0 ? 2 : 0)
         : (kind == kLatFccTrue3 ? (d == 0 ? 2 : 1) : (d < 2 ? 2 : 0));
}
__host__ __device__ constexpr int lat_shell_size(int kind, int k)
{
    return k == 0 ? (kind == kLatBcc ? 8 : 12) : k == 1 ? 6 : (kind == kLatFccTrue3 ? 24 : 12);
}

// The distinct signed axis permutations of shell k's generator, in a fixed order.
struct LatVecs {
    int n;
    int v[24][3];
};
__host__ __device__ constexpr LatVecs lat_vecs(int kind, int k)
{
    LatVecs out{};
    const int perm[6][3] = {{0, 1, 2}, {0, 2, 1}, {1, 0, 2}, {1, 2, 0}, {2, 0, 1}, {2, 1, 0}};
    for (int i = 0; i < 48; ++i) {
        int c[3] = {0, 0, 0};
        for (int d = 0; d < 3; ++d) c[d] = (((i >> (2 - d)) & 1) ? -1 : 1) * lat_gen(kind, k, perm[i >> 3][d]);
        bool dup = false;
        for (int j = 0; j < out.n && !dup; ++j) dup = out.v[j][0] == c[0] && out.v[j][1] == c[1] && out.v[j][2] == c[2];
        if (!dup) {
            for (int d = 0; d < 3; ++d) out.v[out.n][d] = c[d];
            ++out.n;
        }
    }
    return out;
}
// Packed neighbour descriptor for basis b and offset v: (dx+1) | (dy+1) << 2 | (dz+1) << 4 | b' << 6.
__host__ __device__ constexpr int lat_pack(int kind, int b, const int (&v)[3])
{
    int out = 0, par[3] = {0, 0, 0};
    for (int d = 0; d < 3; ++d) {
        const int q = lat_basis(kind, b, d) + v[d];  // -2 .. 3 half units
        par[d] = q & 1;
        out |= ((q >= 0 ? q / 2 : -1) + 1) << (2 * d);
    }
    int bp = 0;
    for (int x = 0; x < lat_nb(kind); ++x)
        if (lat_basis(kind, x, 0) == par[0] && lat_basis(kind, x, 1) == par[1] && lat_basis(kind, x, 2) == par[2])
            bp = x;
    return out | (bp << 6);
}
__host__ __device__ constexpr int lat_desc(int kind, int b, int k, int e) { return lat_pack(kind, b, lat_vecs(kind, k).v[e]); }

// Every descriptor, shells concatenated, for the per-lane lookups of
// lattice_neighbor (a global table: lanes read different entries, which the
// constant bank would serialise).
struct LatDescTable {
    uint8_t d[3][4][54];
};
__host__ __device__ constexpr LatDescTable make_lat_desc_table()
{
    LatDescTable t{};
    for (int kind = 0; kind < 3; ++kind) {
        int e0 = 0;
        for (int k = 0; k < 3; ++k) {
            const LatVecs vs = lat_vecs(kind, k);
            for (int b = 0; b < lat_nb(kind); ++b)
                for (int e = 0; e < vs.n; ++e) t.d[kind][b][e0 + e] = (uint8_t)lat_pack(kind, b, vs.v[e]);
            e0 += vs.n;
        }
    }
    return t;
}
__device__ const LatDescTable kLatDesc = make_lat_desc_table();

// floor(n / d) for 0 <= n < 2^31, d >= 2, from m = floor(2^32 / d): n m / 2^32
// is within n / 2^32 < 1 of n / d, so its floor is the quotient or one less.
__device__ __forceinline__ int div_by(int n, int d, uint32_t m)
{
    int q = (int)__umulhi((uint32_t)n, m);
    q += (n - q * d) >= d;
    return q;
}

struct LatticeCell {
    int b, x, y, z;
};

__device__ __forceinline__ LatticeCell lattice_cell(const LatticeConst &lc, int s)
{
    const int cell = s >> (lc.nb == 4 ? 2 : 1), LL = lc.L * lc.L;  // nb is 2 or 4
    const int x = div_by(cell, LL, lc.mul_LL), r = cell - x * LL, y = div_by(r, lc.L, lc.mul_L);
    return LatticeCell{s & (lc.nb - 1), x, y, r - y * lc.L};
}

// Entry e (shells concatenated) of the neighbour list of the site in cell p.
__device__ __forceinline__ int lattice_neighbor(const LatticeConst &lc, const LatticeCell &p, int e)
{
    const int d = __ldg(&kLatDesc.d[lc.kind][p.b][e]), L = lc.L;
    int x = p.x + (d & 3) - 1, y = p.y + ((d >> 2) & 3) - 1, z = p.z + ((d >> 4) & 3) - 1;
    x += x < 0 ? L : 0;
    y += y < 0 ? L : 0;
    z += z < 0 ? L : 0;
    x -= x >= L ? L : 0;
    y -= y >= L ? L : 0;
    z -= z >= L ? L : 0;
    return lc.nb * ((x * L + y) * L + z) + (d >> 6);
}

// How often s2 is listed in each of the first S shells of s1's neighbour
// list, in closed form: the displacement from s1 to s2 in half units, wrapped
// to (-L, L] per axis, is a shell vector iff its absolute components form the
// shell's pattern (FCC 1,1,0 | 2,0,0 | 2,2,0 or 2,1,1; BCC 1,1,1 | 2,0,0 |
// 2,2,0).  At L = 2 the vectors +2 and -2 along an axis reach the same site,
// so each such component doubles the count.  s1 != s2.
template <int S>
__device__ __forceinline__ void lattice_multiplicity(const LatticeConst &lc, int s1, int s2, uint32_t (&m)[S])
{
    const LatticeCell p = lattice_cell(lc, s1), q = lattice_cell(lc, s2);
    const int M = 2 * lc.L, pc[3] = {p.x, p.y, p.z}, qc[3] = {q.x, q.y, q.z};
    int n0 = 0, n1 = 0, n2 = 0, mult = 1;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        int v = 2 * (qc[d] - pc[d]) + lat_basis(lc.kind, q.b, d) - lat_basis(lc.kind, p.b, d);  // (-2L, 2L)
        v -= v > lc.L ? M : 0;
        v += v <= -lc.L ? M : 0;
        const int a = v < 0 ? -v : v;
        n0 += a == 0;
        n1 += a == 1;
        n2 += a == 2;
        mult <<= (M == 4 && a == 2) ? 1 : 0;
    }
    const bool bcc = lc.kind == kLatBcc, true3 = lc.kind == kLatFccTrue3;
    const bool in[3] = {bcc ? n1 == 3 : (n1 == 2 && n0 == 1), n2 == 1 && n0 == 2,
                        true3 ? (n2 == 1 && n1 == 2) : (n2 == 2 && n0 == 1)};
#pragma unroll
    for (int k = 0; k < S; ++k) m[k] = in[k] ? (uint32_t)mult : 0u;
}

// Compile-time form of the same geometry for the walks over every site
// (recounts): with (kind, b, shell, entry) known at compile time a
// neighbour's id is one sum of three per-site axis terms (LatticeAxes) and b'.
// Per-site axis terms: x[d] = nb L^2 wrap(cx + d - 1), y[d] = nb L wrap(cy + d - 1), z[d] = nb wrap(cz + d - 1).
struct LatticeAxes {
    int x[3], y[3], z[3];
};

__device__ __forceinline__ LatticeAxes lattice_axes(int L, int nb, int cx, int cy, int cz)
{
    const int sx = nb * L * L, sy = nb * L;
    LatticeAxes a;
    a.x[0] = (cx == 0 ? L - 1 : cx - 1) * sx;
    a.x[1] = cx * sx;
    a.x[2] = (cx == L - 1 ? 0 : cx + 1) * sx;
    a.y[0] = (cy == 0 ? L - 1 : cy - 1) * sy;
    a.y[1] = cy * sy;
    a.y[2] = (cy == L - 1 ? 0 : cy + 1) * sy;
    a.z[0] = (cz == 0 ? L - 1 : cz - 1) * nb;
    a.z[1] = cz * nb;
    a.z[2] = (cz == L - 1 ? 0 : cz + 1) * nb;
    return a;
}

template <int D>
__device__ __forceinline__ int lat_id(const LatticeAxes &a)
{
    return a.x[D & 3] + a.y[(D >> 2) & 3] + a.z[(D >> 4) & 3] + (D >> 6);
}

template <int Kind, int B, int K, class H, class W, int... E>
__device__ __forceinline__ H lat_shell_sum(const LatticeAxes &a, W &weight, std::integer_sequence<int, E...>)
{
    return (H(0) + ... + weight(lat_id<lat_desc(Kind, B, K, E)>(a)));
}

// Cells first, first + stride, ... of basis B: site(s, h) with h[k] = sum of
// weight(n) over the shell-k neighbours n of site s.
template <int Kind, int B, int S, class H, class W, class F>
__device__ __forceinline__ void lattice_walk(int L, int first, int stride, W &weight, F &site)
{
    constexpr int NB = lat_nb(Kind);
    const int LL = L * L, ncell = LL * L;
    int cell = first;
    int cx = cell / LL, cy = (cell - cx * LL) / L, cz = cell - cx * LL - cy * L;
    const int bx = stride / LL, by = (stride - bx * LL) / L, bz = stride - bx * LL - by * L;
    for (; cell < ncell; cell += stride) {
        const LatticeAxes a = lattice_axes(L, NB, cx, cy, cz);
        H h[S];
        h[0] = lat_shell_sum<Kind, B, 0, H>(a, weight, std::make_integer_sequence<int, lat_shell_size(Kind, 0)>{});
        if constexpr (S > 1)
            h[1] = lat_shell_sum<Kind, B, 1, H>(a, weight, std::make_integer_sequence<int, lat_shell_size(Kind, 1)>{});
        if constexpr (S > 2)
            h[2] = lat_shell_sum<Kind, B, 2, H>(a, weight, std::make_integer_sequence<int, lat_shell_size(Kind, 2)>{});
        site(NB * cell + B, h);
        cz += bz;  // next cell of the walk: cell += stride in (cx, cy, cz) digits
        if (cz >= L) {
            cz -= L;
            ++cy;
        }
        cy += by;
        if (cy >= L) {
            cy -= L;
            ++cx;
        }
        cx += bx;
    }
}

// Every site of an implicit lattice (this thread's share of a walk that
// starts at cell `first` and steps by `stride` cells, once per basis index, so
// that the threads of a warp share the basis and the neighbour geometry is
// compile-time): site(s, h[S]) with h[k] = sum of weight(n) over the shell-k
// neighbours n of s.
template <int S, class H, class W, class F>
__device__ __forceinline__ void lattice_sites(const LatticeConst &lc, int first, int stride, W weight, F site)
{
    if (lc.kind == kLatBcc) {
        lattice_walk<kLatBcc, 0, S, H>(lc.L, first, stride, weight, site);
        lattice_walk<kLatBcc, 1, S, H>(lc.L, first, stride, weight, site);
    } else if (lc.kind == kLatFccTrue3) {
        lattice_walk<kLatFccTrue3, 0, S, H>(lc.L, first, stride, weight, site);
        lattice_walk<kLatFccTrue3, 1, S, H>(lc.L, first, stride, weight, site);
        lattice_walk<kLatFccTrue3, 2, S, H>(lc.L, first, stride, weight, site);
        lattice_walk<kLatFccTrue3, 3, S, H>(lc.L, first, stride, weight, site);
    } else {
        lattice_walk<kLatFccRef, 0, S, H>(lc.L, first, stride, weight, site);
        lattice_walk<kLatFccRef, 1, S, H>(lc.L, first, stride, weight, site);
        lattice_walk<kLatFccRef, 2, S, H>(lc.L, first, stride, weight, site);
        lattice_walk<kLatFccRef, 3, S, H>(lc.L, first, stride, weight, site);
    }
}

// Shell layout of the padded table, in int4 chunks per shell (0: shell absent).
// Fixed layouts unroll every load; RuntimeShells reads the chunk counts from
// SearchConst; ImplicitShells has no table (neighbours from lattice
// arithmetic), so the search loops of table structures carry no implicit
// code and the other way round.
template <int C0, int C1, int C2>
struct Shells {
    static constexpr int S = (C0 > 0) + (C1 > 0) + (C2 > 0);
    static constexpr bool kRuntime = false;
    static constexpr bool kImplicit = false;
    static constexpr int kRow4 = C0 + C1 + C2;
    __host__ __device__ static constexpr int chunks(int k) { return k == 0 ? C0 : (k == 1 ? C1 : C2); }
    __host__ __device__ static constexpr int off(int k) { return k == 0 ? 0 : (k == 1 ? C0 : C0 + C1); }
};
template <int S_>
struct RuntimeShells {
    static constexpr int S = S_;
    static constexpr bool kRuntime = true;
    static constexpr bool kImplicit = false;
    static constexpr int kRow4 = 0;
    __host__ __device__ static constexpr int chunks(int) { return 0; }
    __host__ __device__ static constexpr int off(int) { return 0; }
};
template <int S_>
struct ImplicitShells {
    static constexpr int S = S_;
    static constexpr bool kRuntime = true;
    static constexpr bool kImplicit = true;
    static constexpr int kRow4 = 0;
    __host__ __device__ static constexpr int chunks(int) { return 0; }
    __host__ __device__ static constexpr int off(int) { return 0; }
};

struct AcceptRecord {
    uint32_t round, task, s1, s2;
    double f2;
};

struct McArgs {
    const int4 *nbor;
    uint8_t *occ;
    int32_t *cnt;
    double *f2;
    uint64_t *hist;           // [slots][N] site histograms (SiteHist)
    const uint32_t *nbmask;   // neighbour-offset bitmap (score_delta)
    const int32_t *order;  // slots searched by this launch, one CTA each
    uint32_t mc_call;
    int32_t tasks, depth;
    int64_t max_rounds;
    unsigned long long *stats;  // [0] rounds, [1] evals, [2] accepts
    // optional trace (tests): per CTA up to trace_cap records and count snapshots
    AcceptRecord *trace;
    int32_t *trace_counts;
    int64_t *trace_len;
    int64_t trace_cap;
    int64_t *rounds_out;  // optional, per CTA
};

struct GenArgs {
    const int4 *nbor;
    uint8_t *occ;
    int32_t *cnt;
    double *f2;
    uint64_t *hist;  // [slots][N] site histograms written by the recount (nullptr: none)
    const int32_t *order;
    uint32_t generation;
    int32_t generate;  // 1: draw a new occupancy; 0: recount the stored one
};

// ---------------------------------------------------------------------------
// Fitness: f2 = sum_k w_k e_k; e_k accumulates d^2 with fma over the upper
// triangle row by row (d_ii, then d_ij and d_ji for j > i); d = fma(-C', R, E).
// Counts are symmetric and R_ij == R_ji, so d_ij and d_ji share C' and R.
// ---------------------------------------------------------------------------
template <int T, int S>
__device__ __forceinline__ double fitness_of_counts(const SearchConst &c, const int32_t *cnt)
{
    double f2 = 0.0;
#pragma unroll
    for (int k = 0; k < S; ++k) {
        double e = 0.0;
#pragma unroll
        for (int i = 0; i < T; ++i) {
            const int ii = (k * T + i) * T + i;
            const double dii = __fma_rn(-(double)cnt[ii], c.R[ii], c.E[ii]);
            e = __fma_rn(dii, dii, e);
#pragma unroll
            for (int j = i + 1; j < T; ++j) {
                const int ij = (k * T + i) * T + j, ji = (k * T + j) * T + i;
                const double cp = (double)cnt[ij];
                const double dij = __fma_rn(-cp, c.R[ij], c.E[ij]);
                const double dji = __fma_rn(-cp, c.R[ij], c.E[ji]);
                e = __fma_rn(dij, dij, e);
                e = __fma_rn(dji, dji, e);
            }
        }
        f2 = __fma_rn(c.w[k], e, f2);
    }
    return f2;
}

// ---------------------------------------------------------------------------
// The swap delta (how proposals are scored).  Swapping species a (at s1) and b
// (at s2) changes the pair counts of shell k by dC_ij = sa_i u_j + sa_j u_i,
// sa = e_a - e_b, where u_t = n2_t - n1_t + m ([t = b] - [t = a]); n1, n2 are
// the species histograms of the two sites' shell-k neighbourhoods and m is how
// often s2 is listed among s1's shell-k neighbours.  dC is zero outside rows and
// columns a, b, so with d = E - R C (R symmetric) the change of
// e_k = sum_ij d_ij^2 is exactly
//     sum_t u_t (L_t + u_t Q_t) + (u_a - u_b)^2 Cq,
//     L_t = -2 (G_at - G_bt),   G_it = R_it (d_it + d_ti),
//     Q_t = 2 (R_at^2 + R_bt^2) for t != a, b,   Q_a = 4 R_aa^2,   Q_b = 4 R_bb^2,
//     Cq  = 2 R_ab^2,
// and f2 changes by D = sum_k w_k (that): O(T) terms per shell instead of the
// O(T^2) of a full fitness.  Fixed operation order (restated by the CPU oracle):
//     Q   = w * (2 * (R_at * R_at + R_bt * R_bt)),  Q_a = w * (4 * (R_aa * R_aa)),
//     Cq  = w * (2 * (R_ab * R_ab)),
//     d_it = fma(-C, R_it, E_it),  G_it = R_it * (d_it + d_ti),  L = (-2 * w) * (G_at - G_bt),
//     D = 0; per shell k: per t < T: D = fma(u_t, fma(u_t, Q_t, L_t), D); then D = fma((u_a - u_b)^2, Cq, D).
// A round's best proposal (lowest D, lowest task on ties) is accepted iff D < 0;
// the search's running f2 adds D, and the f2 a search stores at its end is
// recomputed from the counts (fitness_of_counts).
//
// Which proposal wins is all a round needs of the D's, so they are screened:
// every proposal gets an FP32 value of D and a bound e on its distance from D
// (score_delta), and the FP64 D above is computed (exact_delta) only for those
// whose intervals [D32 - e, D32 + e] leave the winner or its sign open --
// almost always none.  The winner is the same as if all D were compared.
//
// The FP32 table (DeltaTab, shared memory) holds, scaled by a power of two,
// per shell k and ordered pair (a, b) the row of L_t (from the counts, rebuilt
// after every accepted swap) and Q_t, and Cq apart.
//
// The bound: with delta = 2^-24, g_xt = 2 w |G_xt| and A = sum |u_t| (g_at + g_bt),
// the L's are differences of twice rounded g's and all sums together round at most 20
// times, so |D32 - D| <= 24 delta (A + B), B = sum u_t^2 Q_t + sum (u_a - u_b)^2 Cq
// (all positive).  By Cauchy-Schwarz A^2 <= B sum_kt (g_at + g_bt)^2 / Q_t, and
// every (g_at + g_bt)^2 / Q_t is at most 4 max_i w (kappa_it (d_it + d_ti))^2 with
// kappa_it = max(1, n_t / n_i) (it matters for t = a or b, whose Q holds R_tt
// alone).  So e = 32 delta (B + sqrt(B) z), z^2 = 4 S T max_kit w (kappa_it (d_it + d_ti))^2,
// kept with the table; 32 leaves room for the roundings of e itself and of D.
// It holds while the table's values stay in FP32's range, which the host
// checks (SearchConst::screen_floor).
//
// D itself is rounded too.  Where E is symmetric, d_it + d_ti = 2 d_it, rounded
// as the table's one fma rounds it: relative steps of 2^-53, far inside what 32
// leaves over 24.  Else the two differ by up to 2^-52 (|E_it - E_ti| / 2 + C R)
// however small the sum is: by eta R_it, say, which moves D by at most 3 eta B
// (|u| >= 1; the cross terms by Cq and the larger of Q_a, Q_b, since R_aa R_bb =
// R_ab^2).  8 delta B is left for it, so eta <= 2^-23 is covered, which the host
// checks as well; beyond it every D is exact.
// ---------------------------------------------------------------------------
constexpr float kNoSwap = 3.0e38f;  // lo and hi of no proposal, or of one that does not improve
// lo and hi of a warp's record before a pass has found a proposal for it: above every proposal's hi, also where
// all are exact (screen_floor) and hi is 3e38, so that an empty record is never compared with (keep_best)
constexpr float kEmpty = __builtin_huge_valf();
constexpr float kScreenEps = 32.0f / 16777216.0f;

// Layout of the FP32 table, in floats: rows of (k, a, b), within a row species
// t < 2 kPairs in groups {L_t, L_t+1, Q_t, Q_t+1} (one 16-byte load, packed FMAs),
// then {L, Q} of each species left (one or two); Cq [S][T][T]; the coefficients
// of u_a - u_b in the stored u_t, [T][T][kSaRow]; z as found by each warp that
// rebuilds L; the exact D of the accepted swap; and per lane that rebuilds L its
// constants (delta_linear).  Rows are an odd number of 16-byte units apart, which
// spreads lanes' random rows over the banks.
template <int T, int S>
struct DeltaTab {
    static constexpr int kPairs = (T - 1) / 2, kRest = T - 2 * kPairs, kRow = T == 2 ? 4 : 12, kRows = S * T * T;
    static constexpr int kGroups = 32 / T, kWarps = (S * T + kGroups - 1) / kGroups;  // warps that rebuild L
    static constexpr int kSaRow = T == 6 ? 8 : 4;
    static constexpr int kCq = kRows * kRow, kSa = (kCq + kRows + 3) & ~3, kZ = kSa + T * T * kSaRow,
                         kAccepted = kZ + 4, kLanes = kAccepted + 4, kFloats = kLanes + kWarps * 32 * 6;
    static_assert(kWarps <= 4, "one z slot per warp");
    static constexpr float kZScale = S * T <= 4 ? 4.0f : S * T <= 9 ? 6.0f : S * T <= 16 ? 8.0f : 8.5f;  // >= sqrt(4 S T)
    float *f;
    __host__ __device__ static constexpr int lin(int t)
    {
        return t < 2 * kPairs ? 4 * (t / 2) + (t & 1) : 4 * kPairs + 2 * (t - 2 * kPairs);
    }
    __host__ __device__ static constexpr int quad(int t) { return lin(t) + (t < 2 * kPairs ? 2 : 1); }
    __device__ __forceinline__ float *row(int k, int a, int b) const { return f + ((k * T + a) * T + b) * kRow; }
    __device__ __forceinline__ double *accepted() const { return reinterpret_cast<double *>(f + kAccepted); }
    // lane constants of entry i = 32 w + lane: 2 R_xt and E_xt + E_tx; -2 w R_xt and kappa_xt sqrt(w), scaled
    __device__ __forceinline__ double *lane_r2() const { return reinterpret_cast<double *>(f + kLanes); }
    __device__ __forceinline__ double *lane_e() const { return lane_r2() + kWarps * 32; }
    __device__ __forceinline__ float *lane_g() const { return f + kLanes + kWarps * 32 * 4; }
    __device__ __forceinline__ float *lane_z() const { return lane_g() + kWarps * 32; }
};
template <int T>
__host__ __device__ constexpr size_t delta_floats(int S)
{
    return S == 1 ? DeltaTab<T, 1>::kFloats : S == 2 ? DeltaTab<T, 2>::kFloats : DeltaTab<T, 3>::kFloats;
}
__host__ __device__ constexpr size_t delta_bytes(int T, int S)
{
    return sizeof(float) * (T == 2   ? delta_floats<2>(S)
                            : T == 3 ? delta_floats<3>(S)
                            : T == 4 ? delta_floats<4>(S)
                            : T == 5 ? delta_floats<5>(S)
                                     : delta_floats<6>(S));
}

// Q_t of the pair (a, b) in one shell's R, and Cq.
template <int T>
__device__ __forceinline__ double delta_quad(const double *Rk, double w, int a, int b, int t)
{
    if (t == a || t == b) return __dmul_rn(w, __dmul_rn(4.0, __dmul_rn(Rk[t * T + t], Rk[t * T + t])));
    const double p = __dmul_rn(Rk[a * T + t], Rk[a * T + t]), q = __dmul_rn(Rk[b * T + t], Rk[b * T + t]);
    return __dmul_rn(w, __dmul_rn(2.0, __dadd_rn(p, q)));
}
template <int T>
__device__ __forceinline__ double delta_cross(const double *Rk, double w, int a, int b)
{
    return __dmul_rn(w, __dmul_rn(2.0, __dmul_rn(Rk[a * T + b], Rk[a * T + b])));
}

// Structure constants of the table: Q and Cq of every (k, a, b), a != b, the
// coefficients of u_a - u_b, the lanes' constants, and the z slots no warp writes.
// Block-cooperative, no barrier.
template <int T, int S>
__device__ void delta_consts(const SearchConst &c, const DeltaTab<T, S> tab)
{
    using Tab = DeltaTab<T, S>;
    const double scale = c.screen_scale;  // 0: beyond FP32's range, the table is all zero
    for (int e = threadIdx.x; e < S * T * T * T; e += blockDim.x) {
        const int t = e % T, ab = (e / T) % (T * T), k = e / (T * T * T), a = ab / T, b = ab % T;
        if (a == b) continue;
        const double *R = c.R + k * T * T;
        tab.row(k, a, b)[Tab::quad(t)] = scale > 0.0 ? (float)(scale * delta_quad<T>(R, c.w[k], a, b, t)) : 0.0f;
        if (t == 0)
            tab.f[Tab::kCq + k * T * T + ab] = scale > 0.0 ? (float)(scale * delta_cross<T>(R, c.w[k], a, b)) : 0.0f;
        // u of the last species is minus the sum of the others
        if (k == 0 && t < T - 1)
            tab.f[Tab::kSa + ab * Tab::kSaRow + t] =
                (float)((t == a) - (t == b) - (T - 1 == a) + (T - 1 == b));
    }
    for (int i = threadIdx.x; i < 32 * Tab::kWarps; i += blockDim.x) {
        const int x = (i & 31) % T, grp = (i & 31) / T, g = (i >> 5) * Tab::kGroups + grp;
        const bool on = grp < Tab::kGroups && g < S * T;
        const int k = on ? g / T : 0, t = on ? g % T : 0, xt = (k * T + x) * T + t, tx = (k * T + t) * T + x;
        tab.lane_r2()[i] = scale > 0.0 ? 2.0 * c.R[xt] : 0.0;
        tab.lane_e()[i] = scale > 0.0 ? c.E[xt] + c.E[tx] : 0.0;
        tab.lane_g()[i] = scale > 0.0 ? (float)(-2.0 * scale * c.w[k] * c.R[xt]) : 0.0f;
        tab.lane_z()[i] = on && scale > 0.0 ? c.kappa[x * T + t] * c.screen_sw[k] : 0.0f;
    }
    if (threadIdx.x >= Tab::kWarps && threadIdx.x < 4) tab.f[Tab::kZ + threadIdx.x] = 0.0f;
}

// The count-dependent part of the table: L of every row, from the counts
// count_of(k, i, j) (symmetric in i, j), and z; with `cnew`, also stores the
// counts there.  Groups of T lanes of a warp hold G_xt for x = 0..T-1 of one
// (shell, t) -- all (k, x, t) once; each lane takes the others' G by shuffle and
// writes its row x against every y != x.  Warps call it convergently (full-mask
// shuffles, also in count_of); no barrier inside.
//
// It is the longest chain of an accepted round, so the lanes' constants lie in
// shared memory, one conflict-free load each (as indexed loads from the
// kernel's parameters they replayed once per lane).
template <int T, int S, class CountOf>
__device__ __forceinline__ void delta_linear(const DeltaTab<T, S> tab, int32_t *cnew, CountOf count_of)
{
    using Tab = DeltaTab<T, S>;
    const int lane = threadIdx.x & 31, x = lane % T, grp = lane / T;
    for (int w = threadIdx.x >> 5; w < Tab::kWarps; w += blockDim.x >> 5) {
        const int g = w * Tab::kGroups + grp, i = 32 * w + lane;  // shell k = g / T, column t = g % T
        const bool on = grp < Tab::kGroups && g < S * T;
        const int k = on ? g / T : 0, t = on ? g - k * T : 0;
        const int C = count_of(k, x, t);
        if (cnew && on) cnew[(k * T + x) * T + t] = C;
        const float dd = (float)__fma_rn(-(double)C, tab.lane_r2()[i], tab.lane_e()[i]);
        const float G = dd * tab.lane_g()[i], r = dd * tab.lane_z()[i];
        float *row = tab.row(k, x, 0) + Tab::lin(t);
#pragma unroll
        for (int y = 0; y < T; ++y) {
            const float Gy = __shfl_sync(0xFFFFFFFFu, G, lane - x + y);
            if (on && y != x) row[y * Tab::kRow] = G - Gy;
        }
        const float rmax = __uint_as_float(__reduce_max_sync(0xFFFFFFFFu, __float_as_uint(fabsf(r))));
        if (lane == 0) tab.f[Tab::kZ + w] = rmax * Tab::kZScale;
    }
}

// ---------------------------------------------------------------------------
// Site histograms: per slot and site, how many neighbours of each species the
// site has in each shell.  A shell's counts sum to its size, so the last
// species is left out (a difference of two sites' counts of it is minus the
// sum of the others'), and one 64-bit word holds a site: T - 1 fields of 5
// bits per shell (Z <= 28 < 32), shells one after the other, and the site's own
// species in the top 3 bits.  Only six species in three shells need more than
// 64 bits that way: lattice structures then use the 4, 3 and 5 bits that
// their shells of at most 12, 6 and 24 neighbours take, tables of any other
// shells a second word (shell 2 and the species).
//
// Why one word: the two entries of a proposal are random loads, and what they
// cost is set by how much of the population's histograms L2 holds and, beyond
// it, by DRAM's random-access rate.  Measured on B200 from a 4 GiB buffer, 32 CTAs
// of 256 threads per SM: 4.7e10 random 8-byte loads/s (hea_dram_random_probe)
// against 2.3e10 (3.2e10 evict-first) 16-byte ones.
// ---------------------------------------------------------------------------
template <int T, int S, bool kImplicit>
struct SiteHist {
    static constexpr bool kWide = T == 6 && S == 3 && !kImplicit;
    static constexpr bool kTight = T == 6 && S == 3 && kImplicit;
    static constexpr int W = kWide ? 2 : 1;  // 64-bit words per site
    static constexpr int kHalves = 2 * W;    // 32-bit words
    // field (k, t), t < T - 1: its 32-bit word, its place among the word's fields, first bit, width.
    // Uniform: six 5-bit fields per 32-bit word.  Tight: shell 2 then two fields of shell 1 in the
    // low word, shell 0 then the other three of shell 1 in the high word.  Wide: a shell per word.
    __host__ __device__ static constexpr int half(int k, int t)
    {
        return kWide ? k : kTight ? (k == 0 ? 1 : k == 2 ? 0 : t < 2 ? 0 : 1) : (k * (T - 1) + t) / 6;
    }
    __host__ __device__ static constexpr int place(int k, int t)
    {
        return kWide ? t : kTight ? (k != 1 ? t : t < 2 ? 5 + t : 3 + t) : (k * (T - 1) + t) % 6;
    }
    __host__ __device__ static constexpr int width(int k) { return kTight ? (k == 0 ? 4 : k == 1 ? 3 : 5) : 5; }
    __host__ __device__ static constexpr int bit(int k, int t)
    {
        return kTight ? (k == 0 ? 4 * t : k == 2 ? 5 * t : t < 2 ? 25 + 3 * t : 14 + 3 * t) : 5 * place(k, t);
    }
    __host__ __device__ static constexpr int word(int k, int t) { return half(k, t) / 2; }
    __host__ __device__ static constexpr int shift(int k, int t) { return 32 * (half(k, t) & 1) + bit(k, t); }
    // Fields of 32-bit word h at even (odd) places: their mask, and one above each field's top bit
    // (free in that mask), so that differences of all of them take one subtraction.
    __host__ __device__ static constexpr uint32_t fields(int h, int parity)
    {
        uint32_t m = 0;
        for (int k = 0; k < S; ++k)
            for (int t = 0; t < T - 1; ++t)
                if (half(k, t) == h && (place(k, t) & 1) == parity) m |= ((1u << width(k)) - 1u) << bit(k, t);
        return m;
    }
    __host__ __device__ static constexpr uint32_t guards(int h, int parity)
    {
        uint32_t m = 0;
        for (int k = 0; k < S; ++k)
            for (int t = 0; t < T - 1; ++t)
                if (half(k, t) == h && (place(k, t) & 1) == parity) m |= 1u << (bit(k, t) + width(k));
        return m;
    }
};
// Words per site; the host sizes the histogram buffers with it.
__host__ __device__ constexpr int hist_words(int T, int S, bool implicit) { return T == 6 && S == 3 && !implicit ? 2 : 1; }

template <int W>
struct HistEntry {
    uint64_t w[W];
    __device__ __forceinline__ uint32_t half(int h) const { return (uint32_t)(w[h / 2] >> (32 * (h & 1))); }
};

template <class H>
__device__ __forceinline__ int hist_field(const HistEntry<H::W> &e, int k, int t)  // t < T - 1
{
    const uint64_t w = H::W == 1 ? e.w[0] : H::word(k, t) ? e.w[H::W - 1] : e.w[0];  // no indexed array (k, t at run time)
    return (int)((uint32_t)(w >> H::shift(k, t)) & ((1u << H::width(k)) - 1u));
}
template <class H, int T>
__device__ __forceinline__ uint64_t hist_unit(int k, int t)  // one neighbour of species t in shell k
{
    return t < T - 1 ? 1ull << H::shift(k, t) : 0ull;
}
// The site's own species: in six-species three-shell structures the top 3 bits;
// else bits 62 and 63, with bit 31 above them (the uniform fields leave bits 30, 31, 62 and 63 free).
template <class H>
__device__ __forceinline__ int hist_species(const HistEntry<H::W> &e)
{
    const uint64_t w = e.w[H::W - 1];
    if constexpr (H::kWide || H::kTight) return (int)(w >> 61);
    return (int)(w >> 62) | (int)(((uint32_t)w >> 31) << 2);
}
template <class H>
__device__ __forceinline__ uint64_t hist_species_bits(int a)
{
    if constexpr (H::kWide || H::kTight) return (uint64_t)a << 61;
    return ((uint64_t)(a & 3) << 62) | ((uint64_t)(a >> 2) << 31);
}

// Two sites' entries, through L2.  Structures whose histograms are far larger
// than L2 (SearchConst::hist_stream, set by the host) read them evict-first, so
// that random lines from DRAM do not push out those that are read again.
template <int W>
__device__ __forceinline__ void load_hist_pair(const SearchConst &c, const uint64_t *hist, uint32_t s1, uint32_t s2,
                                               HistEntry<W> &p, HistEntry<W> &q)
{
    if constexpr (W == 1) {
        const unsigned long long *h = reinterpret_cast<const unsigned long long *>(hist);
        if (c.hist_stream) {
            p.w[0] = __ldcs(h + s1);
            q.w[0] = __ldcs(h + s2);
        } else {
            p.w[0] = __ldcg(h + s1);
            q.w[0] = __ldcg(h + s2);
        }
    } else {
        const ulonglong2 *h = reinterpret_cast<const ulonglong2 *>(hist);
        const ulonglong2 x = c.hist_stream ? __ldcs(h + s1) : __ldcg(h + s1);
        const ulonglong2 y = c.hist_stream ? __ldcs(h + s2) : __ldcg(h + s2);
        p.w[0] = x.x;
        p.w[1] = x.y;
        q.w[0] = y.x;
        q.w[1] = y.y;
    }
}

__device__ __forceinline__ int count4(const int4 x, uint32_t v)
{
    return ((uint32_t)x.x == v) + ((uint32_t)x.y == v) + ((uint32_t)x.z == v) + ((uint32_t)x.w == v);
}

// d = a * b + c on two floats at once (one instruction on sm_100).
__device__ __forceinline__ float2 ffma2(float2 a, float2 b, float2 c)
{
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;"
        : "=l"(d)
        : "l"(*reinterpret_cast<uint64_t *>(&a)), "l"(*reinterpret_cast<uint64_t *>(&b)),
          "l"(*reinterpret_cast<uint64_t *>(&c)));
    return *reinterpret_cast<float2 *>(&d);
}
__device__ __forceinline__ float2 fmul2(float2 a, float2 b)
{
    uint64_t d;
    asm("mul.rn.f32x2 %0, %1, %2;"
        : "=l"(d)
        : "l"(*reinterpret_cast<uint64_t *>(&a)), "l"(*reinterpret_cast<uint64_t *>(&b)));
    return *reinterpret_cast<float2 *>(&d);
}
__device__ __forceinline__ float2 fadd2(float2 a, float2 b)
{
    uint64_t d;
    asm("add.rn.f32x2 %0, %1, %2;"
        : "=l"(d)
        : "l"(*reinterpret_cast<uint64_t *>(&a)), "l"(*reinterpret_cast<uint64_t *>(&b)));
    return *reinterpret_cast<float2 *>(&d);
}
__device__ __forceinline__ float sqrt_approx(float x)
{
    float r;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// u_t = field_t(q) - field_t(p) of every stored species and shell as floats:
// all differences of a word's even or odd places at once, each biased by its
// guard bit; then each field, where it stands, becomes the low mantissa bits of
// a power of two whose last place is the field's first bit.
template <class H, int T, int S>
__device__ __forceinline__ void hist_diff(const HistEntry<H::W> &p, const HistEntry<H::W> &q, float (&u)[S][T])
{
    uint32_t d[H::kHalves][2];
#pragma unroll
    for (int h = 0; h < H::kHalves; ++h)
#pragma unroll
        for (int y = 0; y < 2; ++y)
            d[h][y] = (q.half(h) & H::fields(h, y)) - (p.half(h) & H::fields(h, y)) + H::guards(h, y);
#pragma unroll
    for (int k = 0; k < S; ++k)
#pragma unroll
        for (int t = 0; t < T - 1; ++t) {
            const uint32_t x = d[H::half(k, t)][H::place(k, t) & 1], field = (2u << H::width(k)) - 1u;
            const int bit = H::bit(k, t), at = bit + H::width(k) + 1 <= 23 ? bit : bit - 20;  // or 20 places down
            u[k][t] = __uint_as_float(((bit == at ? x : x >> 20) & (field << at)) | ((uint32_t)(150 - at) << 23)) -
                      ((float)(1u << (23 - at)) + (float)(1u << H::width(k)));
        }
}

// The FP32 value of one proposal's (scaled) D, and B of its bound: s1 (species
// a, site histograms p), s2 (b, q).  On return p and q have m folded in -- m
// added to field a of p's shell k and to field b of q's -- so that u_t =
// field_t(q) - field_t(p), and u of the last species is minus the sum of the
// others (both totals are Z_k + m); the fields keep their width (n1_a + m <= Z_k
// because s1's list holds s2, of species b, m times; likewise for q).  nbmask has
// bit (n - s + N - 1) set for every table entry n of every site s: a clear bit
// for s2 - s1 proves m = 0 in every shell, a set bit sends the lane to count s2
// in s1's row.
//
// What bounds it: shared-memory wavefronts (lanes read random rows) and issue
// slots.  Per shell of five species: three 16-byte row loads instead of five of
// the FP64 form, packed FMAs, no int-to-double conversions.
template <int T, class L, int W>
__device__ __forceinline__ float score_delta(const SearchConst &c, const int4 *__restrict__ nbor,
                                             const uint32_t *__restrict__ nbmask, const DeltaTab<T, L::S> tab,
                                             HistEntry<W> &p, HistEntry<W> &q, uint32_t s1, uint32_t s2, int a, int b,
                                             float &B)
{
    constexpr int S = L::S;
    using H = SiteHist<T, S, L::kImplicit>;
    using Tab = DeltaTab<T, S>;
    const uint32_t d = s2 - s1 + (uint32_t)c.num_sites - 1u;
    const bool near = (__ldg(nbmask + (d >> 5)) >> (d & 31u)) & 1u;
    if (near) {
        uint32_t m[S];
        if constexpr (L::kImplicit) {
            lattice_multiplicity<S>(c.lat, (int)s1, (int)s2, m);
        } else {
            const int row4 = L::kRuntime ? c.row4 : L::kRow4;
            const int4 *r1 = nbor + (size_t)s1 * row4;
#pragma unroll
            for (int k = 0; k < S; ++k) {
                const int o = L::kRuntime ? c.off4[k] : L::off(k), n = L::kRuntime ? c.chunks[k] : L::chunks(k);
                m[k] = 0;
                for (int ch = 0; ch < n; ++ch) m[k] += count4(__ldg(r1 + o + ch), s2);
            }
        }
#pragma unroll
        for (int k = 0; k < S; ++k) {
#pragma unroll
            for (int x = 0; x < W; ++x) {
                p.w[x] += (W == 1 || H::word(k, 0) == x) ? m[k] * hist_unit<H, T>(k, a) : 0ull;
                q.w[x] += (W == 1 || H::word(k, 0) == x) ? m[k] * hist_unit<H, T>(k, b) : 0ull;
            }
        }
    }
    float u[S][T];
    hist_diff<H, T, S>(p, q, u);
    const float *row = tab.row(0, a, b), *cq = tab.f + Tab::kCq + a * T + b;
    const float4 s4 = *reinterpret_cast<const float4 *>(tab.f + Tab::kSa + (a * T + b) * Tab::kSaRow);
    const float sa[5] = {s4.x, s4.y, s4.z, s4.w, T == 6 ? tab.f[Tab::kSa + (a * T + b) * Tab::kSaRow + 4] : 0.0f};
    float2 lin2 = make_float2(0.0f, 0.0f), quad2 = lin2;
    float lin = 0.0f, quad = 0.0f;
#pragma unroll
    for (int k = 0; k < S; ++k) {
        const float *r = row + k * T * T * Tab::kRow;
        float2 sum2 = make_float2(0.0f, 0.0f), v2 = sum2;  // of the stored u; of sa u: v = u_a - u_b
#pragma unroll
        for (int g = 0; g < Tab::kPairs; ++g) {
            const float4 x = *reinterpret_cast<const float4 *>(r + 4 * g);
            const float2 uu = make_float2(u[k][2 * g], u[k][2 * g + 1]), ss = make_float2(sa[2 * g], sa[2 * g + 1]);
            lin2 = ffma2(uu, make_float2(x.x, x.y), lin2);
            quad2 = ffma2(fmul2(uu, uu), make_float2(x.z, x.w), quad2);
            sum2 = g ? fadd2(sum2, uu) : uu;
            v2 = g ? ffma2(uu, ss, v2) : fmul2(uu, ss);
        }
        float sum = sum2.x + sum2.y, v = v2.x + v2.y;
        if constexpr (Tab::kRest == 2) {
            sum += u[k][T - 2];
            v = fmaf(u[k][T - 2], sa[T - 2], v);
        }
        u[k][T - 1] = -sum;
        if constexpr (Tab::kRest == 2) {
            const float4 x = *reinterpret_cast<const float4 *>(r + 4 * Tab::kPairs);
            lin = fmaf(u[k][T - 2], x.x, lin);
            quad = fmaf(u[k][T - 2] * u[k][T - 2], x.y, quad);
            lin = fmaf(u[k][T - 1], x.z, lin);
            quad = fmaf(u[k][T - 1] * u[k][T - 1], x.w, quad);
        } else {
            const float2 x = *reinterpret_cast<const float2 *>(r + 4 * Tab::kPairs);
            lin = fmaf(u[k][T - 1], x.x, lin);
            quad = fmaf(u[k][T - 1] * u[k][T - 1], x.y, quad);
        }
        quad = fmaf(v * v, cq[k * T * T], quad);
    }
    B = quad + (quad2.x + quad2.y);
    return B + (lin + (lin2.x + lin2.y));
}

// u of a proposal, one per lane: lane k T + t holds u_t of shell k (S T <= 18
// lanes; the others 0).  Convergent warp, p and q the same in every lane.
template <int T, class L, int W>
__device__ __forceinline__ int pair_diff(const HistEntry<W> &p, const HistEntry<W> &q)
{
    constexpr int S = L::S;
    using H = SiteHist<T, S, L::kImplicit>;
    const int lane = threadIdx.x & 31, k = lane / T, t = lane - k * T;
    const bool in = lane < S * T;
    int u = 0;
    if (in && t < T - 1) u = hist_field<H>(q, k, t) - hist_field<H>(p, k, t);
    int rest = 0;
#pragma unroll
    for (int i = 0; i < T - 1; ++i) rest += __shfl_sync(0xFFFFFFFFu, u, in ? k * T + i : 0);
    return in && t == T - 1 ? -rest : u;
}

// D of the proposal (a, b, p, q; the same in every lane, m folded in) exactly
// as the contract orders it, from the counts.  Convergent warp: lane k T + t
// computes the term of species t in shell k, then every lane runs the sum.
template <int T, class L, int W>
__device__ __forceinline__ double exact_delta(const SearchConst &c, const int32_t *cnt, int a, int b, HistEntry<W> p,
                                           HistEntry<W> q)
{
    constexpr int S = L::S;
    const int lane = threadIdx.x & 31;
    const bool in = lane < S * T;
    const int k = in ? lane / T : 0, t = in ? lane - k * T : 0;
    const int u = pair_diff<T, L>(p, q);
    const double *R = c.R + k * T * T, *E = c.E + k * T * T;
    const double Ca = (double)cnt[(k * T + a) * T + t], Cb = (double)cnt[(k * T + b) * T + t];
    const double Ga = __dmul_rn(R[a * T + t], __dadd_rn(__fma_rn(-Ca, R[a * T + t], E[a * T + t]),
                                                         __fma_rn(-Ca, R[a * T + t], E[t * T + a])));
    const double Gb = __dmul_rn(R[b * T + t], __dadd_rn(__fma_rn(-Cb, R[b * T + t], E[b * T + t]),
                                                         __fma_rn(-Cb, R[b * T + t], E[t * T + b])));
    const double lin = __dmul_rn(__dmul_rn(-2.0, c.w[k]), __dsub_rn(Ga, Gb));
    const double inner = __fma_rn((double)u, delta_quad<T>(R, c.w[k], a, b, t), lin);
    double D = 0.0;
#pragma unroll 1
    for (int s = 0; s < S; ++s) {
        for (int i = 0; i < T; ++i)
            D = __fma_rn((double)__shfl_sync(0xFFFFFFFFu, u, s * T + i), __shfl_sync(0xFFFFFFFFu, inner, s * T + i), D);
        const int v = __shfl_sync(0xFFFFFFFFu, u, s * T + a) - __shfl_sync(0xFFFFFFFFu, u, s * T + b);
        D = __fma_rn((double)(v * v), delta_cross<T>(c.R + s * T * T, c.w[s], a, b), D);
    }
    return D;
}

// The same by one lane alone, each of the active lanes with its own proposal.
// Rolled loops: it is rare, and the search loop's code stays small.  Inlined, so
// that its registers are the search loop's (as a call it cost more spills there).
template <int T, class L, int W>
__device__ __forceinline__ double exact_delta_lane(const SearchConst &c, const int32_t *cnt, int ab,
                                                   const HistEntry<W> &p, const HistEntry<W> &q)
{
    constexpr int S = L::S;
    using H = SiteHist<T, S, L::kImplicit>;
    const int a = ab & 0xFF, b = ab >> 8;
    double D = 0.0;
#pragma unroll 1
    for (int k = 0; k < S; ++k) {
        const double *R = c.R + k * T * T, *E = c.E + k * T * T, w = c.w[k];
        int rest = 0, v = 0;
#pragma unroll 1
        for (int t = 0; t < T; ++t) {
            const int u = t < T - 1 ? hist_field<H>(q, k, t) - hist_field<H>(p, k, t) : -rest;
            rest += u;
            v += ((t == a) - (t == b)) * u;
            const double Ra = R[a * T + t], Rb = R[b * T + t];
            const double Ca = (double)cnt[(k * T + a) * T + t], Cb = (double)cnt[(k * T + b) * T + t];
            const double Ga = __dmul_rn(Ra, __dadd_rn(__fma_rn(-Ca, Ra, E[a * T + t]), __fma_rn(-Ca, Ra, E[t * T + a])));
            const double Gb = __dmul_rn(Rb, __dadd_rn(__fma_rn(-Cb, Rb, E[b * T + t]), __fma_rn(-Cb, Rb, E[t * T + b])));
            const double lin = __dmul_rn(__dmul_rn(-2.0, w), __dsub_rn(Ga, Gb));
            D = __fma_rn((double)u, __fma_rn((double)u, delta_quad<T>(R, w, a, b, t), lin), D);
        }
        D = __fma_rn((double)(v * v), delta_cross<T>(R, w, a, b), D);
    }
    return D;
}

// The winner among the warp's candidates whose screened intervals do not
// settle it: the lanes with `in` hold proposals (task, ab = a | b << 8, p, q; m
// folded in).  Proposals of the same species with the same u have the same D (and
// of swapped species with -u: the contract's terms agree bit for bit), so where
// all candidates are such and `negative` says their D < 0, the lowest task wins.
// Few species in few shells (T S <= 6) meet that in most rounds.  Without -> with
// the check, BCC 18^3, 64 solutions x 384 tasks x 4 iterations: T S = 2 0.644 -> 0.629
// ms, 3 0.592 -> 0.567, 2 x 2 0.835 -> 0.775, 4 x 1 0.608 -> 0.597; 6, 8 and 9 level.
// More terms meet it almost never: compiled for all, its code cost the mixed batch
// 7 % (56.5 -> 60.7 ms), so they do without.  Else each candidate computes
// its exact D.  Returns the lane of the lowest D, lowest task on equal D, or -1
// when no D < 0.  Convergent warp.
template <int T, class L, int W>
__device__ __forceinline__ int resolve(const SearchConst &c, const int32_t *cnt, bool in, bool negative, int task,
                                       int ab, const HistEntry<W> &p, const HistEntry<W> &q)
{
    if constexpr (T * L::S <= 6) {
        if (negative) {
            using H = SiteHist<T, L::S, L::kImplicit>;
            const int src = __ffs(__ballot_sync(0xFFFFFFFFu, in)) - 1;
            const bool flip = (ab & 0xFF) > (ab >> 8);
            const int species = flip ? (ab >> 8) | ((ab & 0xFF) << 8) : ab;
            bool same = __shfl_sync(0xFFFFFFFFu, species, src) == species;
#pragma unroll
            for (int h = 0; h < H::kHalves; ++h)
#pragma unroll
                for (int y = 0; y < 2; ++y) {
                    const uint32_t x = q.half(h) & H::fields(h, y), z = p.half(h) & H::fields(h, y);
                    const uint32_t d = flip ? z - x : x - z;  // fields' guard bits keep differences apart
                    same = __shfl_sync(0xFFFFFFFFu, d, src) == d && same;
                }
            if (__all_sync(0xFFFFFFFFu, same || !in)) {
                const uint32_t first = __reduce_min_sync(0xFFFFFFFFu, in ? (uint32_t)task : 0xFFFFFFFFu);
                return __ffs(__ballot_sync(0xFFFFFFFFu, in && (uint32_t)task == first)) - 1;
            }
        }
    }
    uint64_t key = ~0ull;  // ~bits(D) of D < 0: more negative, smaller
    if (in) {
        const double D = exact_delta_lane<T, L, W>(c, cnt, ab, p, q);
        if (D < 0.0) key = ~(uint64_t)__double_as_longlong(D);
    }
    __syncwarp();
    const uint32_t khi = (uint32_t)(key >> 32), klo = (uint32_t)key;
    const uint32_t hi = __reduce_min_sync(0xFFFFFFFFu, khi);
    const uint32_t lo = __reduce_min_sync(0xFFFFFFFFu, khi == hi ? klo : 0xFFFFFFFFu);
    const bool tied = key != ~0ull && khi == hi && klo == lo;
    const uint32_t first = __reduce_min_sync(0xFFFFFFFFu, tied ? (uint32_t)task : 0xFFFFFFFFu);
    return __ffs(__ballot_sync(0xFFFFFFFFu, tied && (uint32_t)task == first)) - 1;
}

// The least float of the warp, as the least of the integers ordered like them.
__device__ __forceinline__ float warp_min(float x)
{
    const int b = __float_as_int(x), m = __reduce_min_sync(0xFFFFFFFFu, b ^ ((b >> 31) & 0x7FFFFFFF));
    return __int_as_float(m ^ ((m >> 31) & 0x7FFFFFFF));
}


// The best of the records lane i < n holds the i-th of (lo, hi: its screened
// interval; load(i): the record): its index, or -1 when none improves.
// Convergent warp.
template <int T, class L, class Load>
__device__ __forceinline__ int best_record(const SearchConst &c, const int32_t *cnt, float lo, float hi, int n,
                                           Load load)
{
    const float least = warp_min(hi);
    const uint32_t cand = __ballot_sync(0xFFFFFFFFu, lo <= least && lo < 0.0f);
    if ((cand & (cand - 1)) == 0 && (cand == 0 || least < 0.0f)) return __ffs(cand) - 1;
    const int lane = threadIdx.x & 31;
    const auto r = load(lane < n ? lane : 0);
    return resolve<T, L>(c, cnt, (cand >> lane) & 1u, least < 0.0f, r.task, r.ab, r.p, r.q);
}

// After an accepted swap of s1 (species a -> b) and s2 (b -> a): update the
// histograms of every neighbour listed in both rows (block-wide, atomics in
// L2; the caller's barrier publishes them).  An entry n in shell k of s1's row
// means s1 is in n's shell k as often, since tables are symmetric per shell.
// Adds of packed fields are exact in any order: the sum is modulo 2^64 and
// every final field is in range.
// kSpecies: also the species bits of s1 and s2, which draw_pair_hist reads;
// searches whose draws read the occupancy leave them at their recount values.
// `me` is this thread's index in the block's order of the work (a rotation of
// threadIdx.x, so that other updates can run on the first warps meanwhile).
template <int T, class L, bool kSpecies>
__device__ __forceinline__ void update_hist(const SearchConst &c, const int4 *__restrict__ nbor, uint64_t *hist,
                                            uint32_t s1, uint32_t s2, int a, int b, int me)
{
    using H = SiteHist<T, L::S, L::kImplicit>;
    unsigned long long *h = reinterpret_cast<unsigned long long *>(hist);
    // one a becomes b among s1's neighbours, one b becomes a among s2's
    const auto add = [h, a, b](int n, int k, bool first) {
        const unsigned long long up = hist_unit<H, T>(k, b) - hist_unit<H, T>(k, a);
        atomicAdd(h + (size_t)n * H::W + H::word(k, 0), first ? up : 0ull - up);
    };
    if constexpr (L::kImplicit) {  // row e of s1 then of s2, shells concatenated
        const int row = c.lat.zoff[L::S - 1] + c.lat.zsize[L::S - 1];
        for (int e = me; e < 2 * row; e += blockDim.x) {
            const bool first = e < row;
            const int idx = first ? e : e - row;
            const int n = lattice_neighbor(c.lat, lattice_cell(c.lat, (int)(first ? s1 : s2)), idx);
            int k = 0;
#pragma unroll
            for (int kk = 1; kk < L::S; ++kk) k += idx >= c.lat.zoff[kk];
            add(n, k, first);
        }
    } else {
        const int row4 = L::kRuntime ? c.row4 : L::kRow4;
        const int row = 4 * row4;
        for (int e = me; e < 2 * row; e += blockDim.x) {
            const bool first = e < row;
            const int idx = first ? e : e - row;
            const int32_t *r = reinterpret_cast<const int32_t *>(nbor + (size_t)(first ? s1 : s2) * row4);
            const int n = __ldg(r + idx);
            if (n >= c.num_sites) continue;  // sentinel padding
            int k = 0;
#pragma unroll
            for (int kk = 1; kk < L::S; ++kk) k += idx >= 4 * (L::kRuntime ? c.off4[kk] : L::off(kk));
            add(n, k, first);
        }
    }
    if (kSpecies && me == 0) {  // adds, since s1 and s2 may be each other's neighbours
        const unsigned long long up = hist_species_bits<H>(b) - hist_species_bits<H>(a);
        atomicAdd(h + (size_t)s1 * H::W + H::W - 1, up);
        atomicAdd(h + (size_t)s2 * H::W + H::W - 1, 0ull - up);
    }
}

// The updates of an accepted swap run on different warps where the block has
// enough of them: counts and table on warps [0, DeltaTab::kWarps), the
// neighbours' histograms on the next.  The rotated thread index keeps the loop
// covering its work once.
__device__ __forceinline__ int block_rotation(int by)
{
    int me = (int)threadIdx.x - by;
    while (me < 0) me += blockDim.x;
    return me;
}

// Attempt j of a Philox call's words: the two sites it draws, and whether both
// draws accept.  Two 32-bit attempts per call, (x0, x1) then (x2, x3); with 16-bit
// draws four, attempt j taking the low and the high half of word x_j (a half in
// the upper 16 bits draws like a 32-bit word: value and remainder of one product).
template <bool k16>
__device__ __forceinline__ bool attempt_sites(const SearchConst &c, const uint32_t (&x)[4], int j, uint32_t &u,
                                              uint32_t &v)
{
    const uint32_t n = (uint32_t)c.num_sites;
    const uint32_t p = k16 ? x[j] << 16 : x[(2 * j) & 3], q = k16 ? x[j] & 0xFFFF0000u : x[(2 * j + 1) & 3];
    u = __umulhi(p, n);
    v = __umulhi(q, n);
    return p * n >= c.reject && q * n >= c.reject;
}

// The first valid attempt from Philox call `call` on: both draws accept and the
// species differ (pyhea/cpp/accelerate.cpp:649-655); differ(u, v) reads them.
template <bool k16, class Differ>
__device__ __forceinline__ bool draw_pair_from(const SearchConst &c, uint32_t call, uint32_t stream, uint32_t round,
                                               uint32_t task, Differ &&differ, uint32_t &s1, uint32_t &s2)
{
    for (; call < kPhiloxCallsPerDraw; ++call) {
        const u32x4 y = philox4x32_10(u32x4{call, task, round, stream}, c.key0, c.key1);
        const uint32_t x[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
        for (int j = 0; j < (k16 ? 4 : 2); ++j) {
            uint32_t u, v;
            if (attempt_sites<k16>(c, x, j, u, v) && differ(u, v)) {
                s1 = u;
                s2 = v;
                return true;
            }
        }
    }
    return false;
}
template <class Differ>
__device__ __forceinline__ bool draw_pair_by(const SearchConst &c, uint32_t stream, uint32_t round, uint32_t task,
                                             Differ &&differ, uint32_t &s1, uint32_t &s2)
{
    return c.draw16 ? draw_pair_from<true>(c, 0, stream, round, task, differ, s1, s2)
                    : draw_pair_from<false>(c, 0, stream, round, task, differ, s1, s2);
}

// All attempts of the first call at once -- the species of every attempt's sites
// in one round trip to shared memory, no branch -- then the calls after it.  A
// warp needs 3 of 4 attempts on average before its last lane has a pair, so the
// loop's dependent loads cost more than the loads left unused (batch of FCC
// 20^3 structures, occupancy in shared memory: 17.4 -> 16.0 ms; in HBM, through
// L1: no difference).
template <bool k16>
__device__ __forceinline__ bool draw_pair_at_once(const SearchConst &c, uint32_t stream, uint32_t round, uint32_t task,
                                                  const uint8_t *occ, uint32_t &s1, uint32_t &s2)
{
    constexpr int A = k16 ? 4 : 2;
    const u32x4 y = philox4x32_10(u32x4{0u, task, round, stream}, c.key0, c.key1);
    const uint32_t x[4] = {y.x, y.y, y.z, y.w};
    uint32_t u[A], v[A];
    bool in[A], ok = false;
#pragma unroll
    for (int j = 0; j < A; ++j) in[j] = attempt_sites<k16>(c, x, j, u[j], v[j]);
#pragma unroll
    for (int j = 0; j < A; ++j) in[j] = (occ[u[j]] != occ[v[j]]) && in[j];
#pragma unroll
    for (int j = A - 1; j >= 0; --j)
        if (in[j]) {
            s1 = u[j];
            s2 = v[j];
            ok = true;
        }
    if (!ok)
        ok = draw_pair_from<k16>(c, 1, stream, round, task,
                                 [occ](uint32_t i, uint32_t j) { return occ[i] != occ[j]; }, s1, s2);
    return ok;
}

// Species from the occupancy.
__device__ __forceinline__ bool draw_pair(const SearchConst &c, uint32_t stream, uint32_t round, uint32_t task,
                                          const uint8_t *occ, uint32_t &s1, uint32_t &s2)
{
    return c.draw16 ? draw_pair_at_once<true>(c, stream, round, task, occ, s1, s2)
                    : draw_pair_at_once<false>(c, stream, round, task, occ, s1, s2);
}

// Species from the site histograms' top bits: for an occupancy in HBM this
// makes the two loads of an attempt the only memory round trip of a proposal;
// p, q are the accepted pair's histograms.
template <class H>
__device__ __forceinline__ bool draw_pair_hist(const SearchConst &c, uint32_t stream, uint32_t round, uint32_t task,
                                               const uint64_t *hist, uint32_t &s1, uint32_t &s2, HistEntry<H::W> &p,
                                               HistEntry<H::W> &q)
{
    return draw_pair_by(
        c, stream, round, task,
        [&c, hist, &p, &q](uint32_t u, uint32_t v) {
            load_hist_pair<H::W>(c, hist, u, v, p, q);
            return hist_species<H>(p) != hist_species<H>(q);
        },
        s1, s2);
}

// A site's histogram entry from its shells' species counts (fields of FB bits,
// one per species, the padding's sentinel entries counted as species 0) and
// its own species a.
template <class H, int T, int S, int FB, class X>
__device__ __forceinline__ HistEntry<H::W> pack_hist(const SearchConst &c, const X (&h)[S], int a)
{
    HistEntry<H::W> e{};
    uint32_t f[H::kHalves] = {};
#pragma unroll
    for (int k = 0; k < S; ++k)
#pragma unroll
        for (int t = 0; t < T - 1; ++t) {
            uint32_t n = (uint32_t)(h[k] >> (FB * t)) & ((1u << FB) - 1u);
            if (t == 0) n -= (uint32_t)c.pad[k];
            f[H::half(k, t)] |= n << H::bit(k, t);
        }
#pragma unroll
    for (int x = 0; x < H::W; ++x) e.w[x] = ((uint64_t)f[2 * x + 1] << 32) | f[2 * x];
    e.w[H::W - 1] |= hist_species_bits<H>(a);
    return e;
}

// ---------------------------------------------------------------------------
// Block recount of the pair counts of the occupancy in shared memory.
// With `hist`, also writes every site's histogram entry (SiteHist).
// Per-thread packed 10-bit accumulators [T][S], flushed to shared-memory bins
// every 32 sites (32 sites * 28 entries < 1024).  Sentinel entries land in
// field 0 and are removed at the end (pad_k * n_i per row i).
// kNeighbors: which neighbour form the caller's structures have, so that a
// kernel compiles the walks it can take.
// ---------------------------------------------------------------------------
enum RecountForm { kRecountTable, kRecountLattice, kRecountEither };

template <int T, int S, RecountForm kNeighbors>
__device__ void block_recount(const SearchConst &c, const int4 *__restrict__ nbor, const uint8_t *occ, int32_t *cnt,
                              uint64_t *hist = nullptr)
{
    for (int x = threadIdx.x; x < S * T * T; x += blockDim.x) cnt[x] = 0;
    __syncthreads();
    uint64_t acc[T][S];
#pragma unroll
    for (int i = 0; i < T; ++i)
#pragma unroll
        for (int k = 0; k < S; ++k) acc[i][k] = 0;
    auto flush = [&]() {
#pragma unroll
        for (int i = 0; i < T; ++i)
#pragma unroll
            for (int k = 0; k < S; ++k) {
#pragma unroll
                for (int t = 0; t < T; ++t) {
                    const int v = (int)((acc[i][k] >> (10 * t)) & 1023u);
                    if (v) atomicAdd(&cnt[(k * T + i) * T + t], v);
                }
                acc[i][k] = 0;
            }
    };
    int since = 0;
    // one site with its shell histograms h (10-bit fields)
    const auto site = [&](int s, const uint64_t (&h)[S], auto form) {
        using H = SiteHist<T, S, decltype(form)::value>;
        const int a = occ[s];
#pragma unroll
        for (int k = 0; k < S; ++k)
#pragma unroll
            for (int i = 0; i < T; ++i)
                if (a == i) acc[i][k] += h[k];
        if (hist) {
            const HistEntry<H::W> e = pack_hist<H, T, S, 10>(c, h, a);
#pragma unroll
            for (int x = 0; x < H::W; ++x) hist[(size_t)s * H::W + x] = e.w[x];
        }
        if (++since == 32) {
            flush();
            since = 0;
        }
    };
    if (kNeighbors == kRecountLattice || (kNeighbors == kRecountEither && c.lat.L)) {
        // implicit neighbours (no sentinel padding: pad[k] == 0)
        if constexpr (kNeighbors != kRecountTable)
            lattice_sites<S, uint64_t>(c.lat, threadIdx.x, blockDim.x,
                                       [occ](int n) { return 1ull << (10 * occ[n]); },
                                       [&site](int s, const uint64_t (&h)[S]) { site(s, h, std::true_type{}); });
    } else if constexpr (kNeighbors != kRecountLattice) {
        for (int s = threadIdx.x; s < c.num_sites; s += blockDim.x) {
            uint64_t h[S];
#pragma unroll
            for (int k = 0; k < S; ++k) {
                h[k] = 0;
                const int4 *seg = nbor + (size_t)s * c.row4 + c.off4[k];
                for (int ch = 0; ch < c.chunks[k]; ++ch) {
                    const int4 x = __ldg(seg + ch);
                    h[k] += (1ull << (10 * occ[x.x])) + (1ull << (10 * occ[x.y])) + (1ull << (10 * occ[x.z])) +
                            (1ull << (10 * occ[x.w]));
                }
            }
            site(s, h, std::false_type{});
        }
    }
    flush();
    __syncthreads();
    for (int x = threadIdx.x; x < S * T; x += blockDim.x) {
        const int k = x / T, i = x % T;
        cnt[(k * T + i) * T] -= c.pad[k] * (c.prefix[i + 1] - c.prefix[i]);
    }
    __syncthreads();
}

// ---------------------------------------------------------------------------
// Random occupancy of population position `pos` of generation `generation`:
// the sorted species layout read through a keyed Feistel permutation (cycle
// walking).  Writes the species into occ and, when gocc != nullptr, also into
// the slot's row in HBM.  Block-cooperative; no barrier inside.
// ---------------------------------------------------------------------------
template <int T>
__device__ __forceinline__ void generate_occupancy(const SearchConst &c, uint32_t pos, uint32_t generation,
                                                   uint8_t *occ, uint8_t *gocc)
{
    uint32_t rk[kFeistelRounds];
    const u32x4 w0 = philox4x32_10(u32x4{pos, generation, 0u, kInitStream}, c.key0, c.key1);
    const u32x4 w1 = philox4x32_10(u32x4{pos, generation, 1u, kInitStream}, c.key0, c.key1);
    rk[0] = w0.x; rk[1] = w0.y; rk[2] = w0.z; rk[3] = w0.w; rk[4] = w1.x; rk[5] = w1.y;
    const int n = c.num_sites;
    for (int s = threadIdx.x; s < n; s += blockDim.x) {
        uint32_t y = feistel((uint32_t)s, c.feistel_h, rk);
        while (y >= (uint32_t)n) y = feistel(y, c.feistel_h, rk);
        int t = 0;
#pragma unroll
        for (int i = 1; i < T; ++i) t += (int)(y >= (uint32_t)c.prefix[i]);
        occ[s] = (uint8_t)t;
        if (gocc) gocc[s] = (uint8_t)t;
    }
}

// New random occupancy or a recount of a stored one; writes occupancy, counts
// and f2 of the slot.  One CTA per slot; dynamic shared memory = occ_stride +
// 16 + 4*S*T*T bytes.
template <int T, int S>
__global__ void __launch_bounds__(512, 1) generate_kernel(const SearchConst c, const GenArgs g)
{
    extern __shared__ __align__(16) uint8_t smem[];
    uint8_t *occ = smem;
    int32_t *cnt = reinterpret_cast<int32_t *>(smem + c.occ_stride + 16);
    const int slot = g.order[blockIdx.x];
    uint8_t *gocc = g.occ + (size_t)slot * c.occ_stride;
    const int n = c.num_sites;
    if (g.generate) {
        generate_occupancy<T>(c, blockIdx.x, g.generation, occ, gocc);
    } else {
        for (int s = threadIdx.x; s < n; s += blockDim.x) occ[s] = gocc[s];
    }
    if (threadIdx.x == 0) occ[n] = 0;
    __syncthreads();
    block_recount<T, S, kRecountEither>(c, g.nbor, occ, cnt,
                                        g.hist ? g.hist + (size_t)slot * n * hist_words(T, S, c.lat.L > 0) : nullptr);
    int32_t *gc = g.cnt + (size_t)slot * S * T * T;
    for (int x = threadIdx.x; x < S * T * T; x += blockDim.x) gc[x] = cnt[x];
    if (threadIdx.x == 0) g.f2[slot] = fitness_of_counts<T, S>(c, cnt);
}

// ---------------------------------------------------------------------------
// The local parallel search (pyhea/cpp/accelerate.cpp:601-694): one CTA per
// solution, one lane per task (lanes loop when tasks > blockDim).  Each round
// every task scores one proposal against the same state (its delta D,
// screened: see score_delta); the block takes the (D, task) minimum and accepts
// it iff D < 0; the search ends after `depth` rounds in a row without an accept.
//
// One block barrier per round: each warp publishes its best proposal (a
// SwapRecord, double-buffered by round parity) before the barrier; after it
// every warp reduces the records itself and writes the winning swap into the
// occupancy (all threads write the same two bytes).  On an accept the block
// writes the counts after the swap into the other count buffer, rebuilds the
// table's L from them and updates the site histograms; a second barrier
// publishes all three before the next round.
//
// Shared memory after the occupancy: the delta table, the records, two count
// buffers (search_smem_tail).
// ---------------------------------------------------------------------------
template <int W>
struct __align__(16) SwapRecord {
    float lo, hi;       // the proposal's D is in [lo, hi] (scaled); kNoSwap when there is none
    int32_t task;
    uint32_t s1, s2;
    int32_t ab;         // species a | b << 8 before the swap
    HistEntry<W> p, q;  // histograms of both sites, m folded in (score_delta)
    int32_t stop;       // record 0 of a round: the block stops after it (deadline)
    int32_t pad_;
};
static_assert(sizeof(SwapRecord<1>) == 48 && sizeof(SwapRecord<2>) == 64, "SwapRecord layout");
// Bytes of a record for either neighbour form.
__host__ __device__ constexpr size_t record_bytes(int T, int S) { return hist_words(T, S, false) == 2 ? 64 : 48; }

__host__ __device__ constexpr int mc_ncount_pad(int ncount) { return (ncount + 3) & ~3; }

// Shared-memory bytes of a search after its occupancy: delta table, 2 * nwarps
// swap records, two count buffers.
__host__ __device__ constexpr size_t search_smem_tail(int T, int S, int nwarps)
{
    return delta_bytes(T, S) + (size_t)2 * nwarps * record_bytes(T, S) +
           (size_t)2 * 4 * mc_ncount_pad(S * T * T);
}

// [lo, hi] of a proposal's D from its screened value and B; both kNoSwap when
// there is no proposal or its D >= 0 for certain.
template <int T, int S>
__device__ __forceinline__ void screen_interval(const SearchConst &c, const DeltaTab<T, S> tab, bool ok, float D,
                                                float B, float &lo, float &hi)
{
    const float4 z4 = *reinterpret_cast<const float4 *>(tab.f + DeltaTab<T, S>::kZ);
    const float z = fmaxf(fmaxf(z4.x, z4.y), fmaxf(z4.z, z4.w));
    const float e = fmaf(kScreenEps, fmaf(sqrt_approx(B), z, B), c.screen_floor);
    ok = ok && D < e;
    lo = ok ? D - e : kNoSwap;
    hi = ok ? D + e : kNoSwap;
}

// Folds the warp's proposals of one pass (lane: r) into its best record of the
// round, `mine` (in shared memory; `more`: it may hold an earlier pass's).
// Convergent warp.
template <int T, class L, class Record>
__device__ __forceinline__ void keep_best(const SearchConst &c, const int32_t *cnt, Record &mine, const Record &r,
                                          bool more)
{
    const float least = warp_min(r.hi);
    const uint32_t cand = __ballot_sync(0xFFFFFFFFu, r.lo <= least && r.lo < 0.0f);
    if (cand) {
        const int lane = threadIdx.x & 31;
        int win = __ffs(cand) - 1;
        if (cand & (cand - 1)) win = resolve<T, L>(c, cnt, (cand >> lane) & 1u, least < 0.0f, r.task, r.ab, r.p, r.q);
        if (lane == win) {
            bool take = !more || r.hi < mine.lo;  // mine.lo = kEmpty: no pass before found a D < 0
            if (!take && r.lo <= mine.hi) {  // an earlier pass's best too near to tell; on equal D it has the lower task
                double before = 0.0, D = 0.0;
#pragma unroll 1
                for (int x = 0; x < 2; ++x) {
                    auto p = r.p, q = r.q;
                    int ab = r.ab;
                    if (x == 0) {
                        p = mine.p;
                        q = mine.q;
                        ab = mine.ab;
                    }
                    before = D;
                    D = exact_delta_lane<T, L>(c, cnt, ab, p, q);
                }
                take = D < before;
            }
            if (take) mine = r;
        }
    }
    __syncwarp();
}

struct McTrace {
    AcceptRecord *records;  // trace_cap records for this search, or nullptr
    int32_t *counts;        // trace_cap count snapshots, or nullptr
    int64_t cap;
};

struct McTally {
    double f2;  // recomputed from the counts, or the running f2 of a yielded search with a tolerance
    int64_t rounds, accepts, evals;  // rounds run by this call
    int64_t round_end;               // round index the search continues from
    int miss;                        // consecutive rejections at round_end
    int buf;                         // count buffer holding the final counts
    bool yielded;                    // stopped at the deadline before converging
};

// Where a search segment starts: a search stopped at a round boundary
// continues from (round0, miss0) with the same occupancy, counts and running
// f2 and draws the same proposals as one that never stopped.
struct McResume {
    int64_t round0;
    int miss0;
    unsigned long long deadline_ns;  // kYield: stop after the first round ending past this device time (0: never)
    double tol2;                     // kYield: the search ends once its running f2 <= tol2 (< 0: never)
};

// Count change dC_ij of shell k for a swap of species a and b with the lanes'
// u of pair_diff: sa_i u_j + sa_j u_i.  Convergent warp.
template <int T>
__device__ __forceinline__ int count_change(int u, int a, int b, int k, int i, int j)
{
    const int ui = __shfl_sync(0xFFFFFFFFu, u, k * T + i), uj = __shfl_sync(0xFFFFFFFFu, u, k * T + j);
    return ((i == a) - (i == b)) * uj + ((j == a) - (j == b)) * ui;
}

// The accept's new counts and L of the table, on the block's first warps
// (DeltaTab::kWarps).
template <int T, class L, class R>
__device__ __forceinline__ void accept_counts(const DeltaTab<T, L::S> tab, const R &w, int a, int b,
                                              const int32_t *cold, int32_t *cnew)
{
    using Tab = DeltaTab<T, L::S>;
    if ((int)(threadIdx.x >> 5) >= Tab::kWarps) return;
    const int u = pair_diff<T, L>(w.p, w.q);
    delta_linear<T, L::S>(tab, cnew, [cold, u, a, b](int k, int i, int j) {
        return cold[(k * T + i) * T + j] + count_change<T>(u, a, b, k, i, j);
    });
}

// Delta table of a search starting from the counts in buffer 0 of cnt2
// Block-wide.
template <int T, int S>
__device__ __forceinline__ void search_setup(const SearchConst &c, const int32_t *cnt2, const DeltaTab<T, S> tab)
{
    delta_consts<T, S>(c, tab);
    __syncthreads();  // the lanes' constants
    delta_linear<T, S>(tab, nullptr, [cnt2](int k, int i, int j) { return cnt2[(k * T + i) * T + j]; });
    __syncthreads();
}

// Rounds of the local search on the staged state: occupancy occ, counts in
// buffer 0 of cnt2, the delta table tab (search_setup), running f2 `cur`.
// Every thread returns the same tally; evals is this thread's count.  No
// barrier at entry.  occ is in shared or global memory.  The
// draws read the species from occ; proposals are scored from the
// site histograms `hist`, which an accept updates.
template <int T, class L, bool kYield = false>
__device__ __forceinline__ McTally mc_rounds(const SearchConst &c, const int4 *__restrict__ nbor, uint8_t *occ,
                                             int32_t *cnt2, const DeltaTab<T, L::S> tab, void *records, uint32_t stream,
                                             double cur, int tasks, int depth, int64_t max_rounds, McTrace tr,
                                             McResume rs, uint64_t *hist, const uint32_t *nbmask)
{
    constexpr int S = L::S, NC = S * T * T, NCP = mc_ncount_pad(NC);
    constexpr int W = SiteHist<T, S, L::kImplicit>::W;
    using Record = SwapRecord<W>;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
    Record *rec = static_cast<Record *>(records);  // [2][nwarps]
    int miss = rs.miss0, buf = 0;
    int64_t round = rs.round0, accepts = 0;
    uint32_t undrawn = 0;  // this thread's tasks that found no pair
    bool yielded = false;
    // the running f2 adds exact D's; nothing else needs them
    const bool track = tr.records || (kYield && rs.tol2 >= 0.0);
    while (miss < depth && round < max_rounds && !(kYield && cur <= rs.tol2)) {
        Record *rr = rec + (round & 1) * nwarps;
        Record &mine = rr[warp];  // this warp's best proposal of the round
        if (lane == 0) mine.lo = mine.hi = kEmpty;
        __syncwarp();
        const int32_t *cold = cnt2 + buf * NCP;
        // passes of blockDim tasks; lane q of a pass scores task q (warp-uniform trip count)
        for (int q0 = warp * 32; q0 < tasks; q0 += blockDim.x) {
            const int q = q0 + lane;
            uint32_t s1 = 0, s2 = 0;  // a lane without a pair scores site 0 with itself and drops the result
            const bool ok = q < tasks && draw_pair(c, stream, (uint32_t)round, (uint32_t)q, occ, s1, s2);
            __syncwarp();  // lanes that needed more draws rejoin before scoring
            undrawn += q < tasks && !ok;
            Record r;
            load_hist_pair<W>(c, hist, s1, s2, r.p, r.q);
            const int a = occ[s1], b = occ[s2];
            r.ab = a | (b << 8);
            float B;
            const float D = score_delta<T, L>(c, nbor, nbmask, tab, r.p, r.q, s1, s2, a, b, B);
            screen_interval(c, tab, ok, D, B, r.lo, r.hi);
            r.task = q;
            r.s1 = s1;
            r.s2 = s2;
            r.stop = 0;
            r.pad_ = 0;
            keep_best<T, L>(c, cold, mine, r, q0 != warp * 32);
        }
        // the stop decision travels in warp 0's record (read by all after the barrier)
        if (kYield && tid == 0) rr[0].stop = (rs.deadline_ns && global_ns() >= rs.deadline_ns) ? 1 : 0;
        __syncwarp();
        __syncthreads();
        const bool stop = kYield && rr[0].stop != 0;
        // every warp reduces the records of all warps
        const int xw = best_record<T, L>(c, cold, lane < nwarps ? rr[lane].lo : kNoSwap,
                                         lane < nwarps ? rr[lane].hi : kNoSwap, nwarps,
                                         [rr](int i) -> const Record & { return rr[i]; });
        if (xw >= 0) {
            const Record &w = rr[xw];
            const int a = w.ab & 0xFF, b = w.ab >> 8;
            if (tid == 0) {  // read again only after the barrier below
                occ[w.s1] = (uint8_t)b;
                occ[w.s2] = (uint8_t)a;
            }
            int32_t *cnew = cnt2 + (buf ^ 1) * NCP;
            accept_counts<T, L>(tab, w, a, b, cold, cnew);
            update_hist<T, L, false>(c, nbor, hist, w.s1, w.s2, a, b, block_rotation(32 * DeltaTab<T, S>::kWarps));
            if (track && warp == nwarps - 1) {
                const double D = exact_delta<T, L>(c, cold, a, b, w.p, w.q);
                if (lane == 0) *tab.accepted() = D;
            }
            __syncwarp();
            __syncthreads();  // next round's proposals read the new table and histograms
            buf ^= 1;
            if (track) cur = __dadd_rn(cur, *tab.accepted());
            if (tr.records && warp == 0 && accepts < tr.cap) {
                if (lane == 0) {
                    AcceptRecord r;
                    r.round = (uint32_t)round;
                    r.task = (uint32_t)rr[xw].task;
                    r.s1 = rr[xw].s1;
                    r.s2 = rr[xw].s2;
                    r.f2 = cur;
                    tr.records[accepts] = r;
                }
                if (tr.counts) {
                    int32_t *dst = tr.counts + accepts * NC;
                    for (int x = lane; x < NC; x += 32) dst[x] = cnew[x];
                }
            }
            miss = 0;
            ++accepts;
        } else {
            ++miss;
        }
        ++round;
        if (kYield && stop && miss < depth && round < max_rounds && !(cur <= rs.tol2)) {
            yielded = true;
            break;
        }
    }
    __syncthreads();
    const int64_t scored = (int64_t)(tid < tasks ? (tasks - 1 - tid) / (int)blockDim.x + 1 : 0) * (round - rs.round0);
    const int64_t evals = scored - undrawn;
    const double f2 = yielded && track ? cur : fitness_of_counts<T, S>(c, cnt2 + buf * NCP);
    return McTally{f2, round - rs.round0, accepts, evals, round, miss, buf, yielded};
}

// One occupancy row to another (16-byte vectors).  kFromL2: load through L2 only
// (rows written earlier by other CTAs of the same launch may sit stale in this
// SM's L1); a row copied onto itself that way is fresh in L1 afterwards.
template <bool kFromL2 = false>
__device__ __forceinline__ void copy_occupancy(const SearchConst &c, const uint8_t *from, uint8_t *to)
{
    const uint4 *src = reinterpret_cast<const uint4 *>(from);
    uint4 *dst = reinterpret_cast<uint4 *>(to);
    for (int v = threadIdx.x; v < c.occ_stride / 16; v += blockDim.x) dst[v] = kFromL2 ? __ldcg(src + v) : src[v];
}

// Sum of per-thread evaluation counts of the block, added to stats[1];
// rounds and accepts (uniform) to stats[0] and stats[2] by thread 0.
__device__ __forceinline__ void add_tally(const McTally &t, unsigned long long *stats)
{
    unsigned long long ev = (unsigned long long)t.evals;
#pragma unroll
    for (int o = 16; o; o >>= 1) ev += __shfl_xor_sync(0xFFFFFFFFu, ev, o);
    if ((threadIdx.x & 31) == 0 && ev) atomicAdd(&stats[1], ev);
    if (threadIdx.x == 0) {
        atomicAdd(&stats[0], (unsigned long long)t.rounds);
        atomicAdd(&stats[2], (unsigned long long)t.accepts);
    }
}

#ifndef HEA_MC_MIN_BLOCKS
#define HEA_MC_MIN_BLOCKS 2  // resident 512-thread blocks per SM the register budget aims for
#endif
// Shared memory: occ_stride + 16 + search_smem_tail(T, S, nwarps).
template <int T, class L>
__global__ void __launch_bounds__(512, HEA_MC_MIN_BLOCKS) mc_kernel(const __grid_constant__ SearchConst c,
                                                                               const McArgs g)
{
    constexpr int S = L::S, NC = S * T * T, NCP = mc_ncount_pad(NC);
    extern __shared__ __align__(16) uint8_t smem[];
    const int tid = threadIdx.x, nwarps = blockDim.x >> 5;
    uint8_t *occ = smem;
    const DeltaTab<T, S> tab{reinterpret_cast<float *>(smem + c.occ_stride + 16)};
    uint8_t *rec = reinterpret_cast<uint8_t *>(tab.f + DeltaTab<T, S>::kFloats);         // [2][nwarps] records
    int32_t *cnt2 = reinterpret_cast<int32_t *>(rec + 2 * nwarps * record_bytes(T, S));  // [2][NCP]

    const int slot = g.order[blockIdx.x];
    const uint32_t stream = (g.mc_call << 16) | (uint32_t)blockIdx.x;
    uint8_t *gocc = g.occ + (size_t)slot * c.occ_stride;
    int32_t *gcnt = g.cnt + (size_t)slot * NC;

    copy_occupancy(c, gocc, occ);
    for (int x = tid; x < NC; x += blockDim.x) cnt2[x] = gcnt[x];
    __syncthreads();
    if (tid == 0) occ[c.num_sites] = 0;  // sentinel (occ_stride may end exactly at n)
    search_setup<T, S>(c, cnt2, tab);

    McTrace tr{nullptr, nullptr, 0};
    if (g.trace) {
        tr.records = g.trace + (size_t)blockIdx.x * g.trace_cap;
        tr.counts = g.trace_counts ? g.trace_counts + (size_t)blockIdx.x * g.trace_cap * NC : nullptr;
        tr.cap = g.trace_cap;
    }
    const McTally t = mc_rounds<T, L>(c, g.nbor, occ, cnt2, tab, rec, stream, g.f2[slot], g.tasks, g.depth,
                                      g.max_rounds, tr, McResume{0, 0, 0ull, -1.0},
                                      g.hist + (size_t)slot * c.num_sites * hist_words(T, S, L::kImplicit),
                                      g.nbmask);

    copy_occupancy(c, occ, gocc);
    for (int x = tid; x < NC; x += blockDim.x) gcnt[x] = cnt2[t.buf * NCP + x];
    add_tally(t, g.stats);
    if (tid == 0) {
        g.f2[slot] = t.f2;
        if (g.trace_len) g.trace_len[blockIdx.x] = t.accepts;
        if (g.rounds_out) g.rounds_out[blockIdx.x] = t.rounds;
    }
}

}  // namespace hea
