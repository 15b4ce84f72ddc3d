// D_mumu / <dmu^2> lag-pair statistics on the device
// (process_mu_chunk_dmumu_cpu!, src/compute_delta_mu2_dmumu_full.jl:457-704).
//
// Sliding estimator (dmumu_kernel)
// --------------------------------
// A particle slot of a CTA stages one particle's mu series in shared memory
// with the list of its starts grouped by start bin; the warps of the slot then
// share the list.  A warp covers 8 lag sets of 8 lags (NS sets, as many as the
// lags need): lane = (start j = 0..3) x (lag l = 0..7), so a row of the pair
// loop is 4 starts of one bin against 8 lags of one set, and every lane keeps
// (sum dmu, sum dmu^2) of its NS lags for the current bin in registers.  At the
// end of a bin the four starts' sums are added across lanes and flushed to the
// CTA's (bin, lag) partials.  Compared with one lag per lane: 55 lags fill 56
// of 56 lane columns instead of 55 of 64, and the start's index, value and
// float-to-double conversion are shared by all NS sets.
//
// No pair is tested for NaN when the particle's finite saves are a prefix
// [0, nfin) of its series (all of it, or the saves until it left an open box):
// a pair is then valid exactly when s + L < nfin, one predicate on the address,
// and the pair counts need no work in the pair loop at all -- a start adds one
// to hist2[bin][k], k = the number of lags it can reach, and the suffix sums of
// hist2 over k are the counts.  Other particles take a loop that tests the
// partner and counts pairs.
//
// What bounds it: instruction issue (63 % busy at 16 warps per SM) with the
// shared-memory pipe (69 %) and the conversion pipe (50 %) close behind; a pair
// row costs an address add, a load, a conversion, two adds and an FMA.  131,072
// x 4001 saves x 55 lags x 50 bins: 28.2 ms with one lag per lane, 15.1 ms now
// (1.6e12 pairs/s); 4096 x 801 x 19 x 20: 263 us, 147 us now.
//
// Injection estimator (dmumu_injection_kernel): only saves 0 and the lags are
// read: 524,287 particles x 29 of 801 saves take 139 us; staging every save as
// the sliding estimator must took 3.7 ms.
//
// CTA results go to per-CTA partials; a finalize kernel adds them in a fixed
// order and merges Welford triples with the reference formula
// (combine_welford_stats!, :439-455).  Integer counts are exact; FP64 sums
// differ from the reference only by summation order.
#include <math_constants.h>

#include <algorithm>
#include <cfloat>
#include <mutex>
#include <type_traits>

#include "pt_internal.cuh"

namespace pt {
namespace {

constexpr int kWarp = 32;
constexpr int kLagLanes = 8;    // lags of a set: lanes of a row along the lag axis
constexpr int kStartLanes = 4;  // starts of a row
constexpr int kMaxSets = 8;     // lag sets of a warp (64 lags)
// Threads of a CTA: the accumulators of NS sets decide the registers of a thread.
// 7 sets, 131,072 x 4001 saves: 15.1 ms with 512 threads, 18.1 with 384, 21.3 with
// 640 (96 registers, spilled); 4 sets, 65,536 x 801: 1.33 ms with 512, 1.25 with 640,
// 1.40 with 768.
__host__ __device__ constexpr int max_threads(int ns) { return ns <= 4 ? 640 : 512; }
constexpr int kBatch = 4;       // saves that a thread stages side by side
constexpr int kKeep = 16;       // saves per thread whose bucket and rank stay in registers until the list is written
constexpr int kFlushCost = 28;  // starts whose pairs cost as much as the end of a bin, its last rows included
constexpr int kMaxSlots = 15;   // one named barrier per slot (barrier 0 is __syncthreads)

struct WelfordPart {
    long long count;
    double mean, m2, pair_ss;
    long long pair_n;
};

// combine_welford_stats! (src/compute_delta_mu2_dmumu_full.jl:439-455)
__device__ __forceinline__ void welford_merge(long long& gc, double& gm, double& gm2, long long lc, double lm,
                                              double lm2)
{
    if (lc <= 0) return;
    if (gc == 0) {
        gc = lc; gm = lm; gm2 = lm2;
        return;
    }
    const long long cc = gc + lc;
    const double delta = lm - gm, share = (double)lc / (double)cc;
    gm += delta * share;
    gm2 += lm2 + delta * delta * (double)gc * share;
    gc = cc;
}

// Bin edges at the series' precision.  mu is compared with the stored Float64
// edges; for a Float32 mu, edge <= mu is the same as (edge rounded up to
// Float32) <= mu, and mu > edge the same as mu > (edge rounded down).  A first edge
// of -Inf becomes the lowest finite value: the same for every finite mu, and a mu of
// -Inf, which has no bin, fails the comparison that bins_of makes first.
__device__ __forceinline__ float edge_up(double e, float)
{
    return e == -CUDART_INF ? -FLT_MAX : __double2float_ru(e);
}
__device__ __forceinline__ double edge_up(double e, double) { return e == -CUDART_INF ? -DBL_MAX : e; }
__device__ __forceinline__ float edge_down(double e, float) { return __double2float_rd(e); }
__device__ __forceinline__ double edge_down(double e, double) { return e; }

template <typename MuT>
struct BinEdges {
    const MuT* up;  // [n_bins + 1] edges rounded up
    MuT first;      // up[0]
    MuT last;       // edges[n_bins] rounded down
    MuT inv_w;      // n_bins / (edges[n_bins] - edges[0])
    int n_bins, bin_abs;
};

// mu_bin_value + mu_bin_index_full (dmumu:304-318) of a finite value: 0-based
// bin, n_bins outside [edges[0], edges[n_bins]].  searchsortedlast (the last
// edge <= v) is found from a guess on a uniform grid, moved up and down until
// edges[b] <= v < edges[b + 1]: the same bin as a binary search for any
// increasing edges.
template <typename MuT>
__device__ __noinline__ int bin_walk(MuT v, const MuT* up, MuT last, int n_bins, int b)
{
    if (v < up[0] || v > last) return n_bins;
    while (b < n_bins && up[b + 1] <= v) ++b;
    while (b > 0 && up[b] > v) --b;
    return b == n_bins ? n_bins - 1 : b;  // v == edges[n_bins] falls in the last bin
}

// Bins of N values (-1: not finite), the guesses side by side: the uniform edges
// of build_mu_edges_full confirm them with two compares, and only values on an
// edge, outside, or between uneven edges walk.
template <int N, typename MuT>
__device__ __forceinline__ void bins_of(const MuT (&v)[N], const BinEdges<MuT>& E, int (&b)[N])
{
    bool walk[N], any = false;
#pragma unroll
    for (int i = 0; i < N; ++i) {
        const MuT t = E.bin_abs ? fabs(v[i]) : v[i];
        const int g = (int)fmin(fmax((t - E.first) * E.inv_w, MuT(0)), (MuT)(E.n_bins - 1));
        walk[i] = !(E.up[g] <= t && t < E.up[g + 1]);
        b[i] = g;
        any |= walk[i];
    }
    if (any) {
#pragma unroll
        for (int i = 0; i < N; ++i)
            if (walk[i])
                b[i] = fabs(v[i]) < MuT(CUDART_INF)
                           ? bin_walk(E.bin_abs ? (MuT)fabs(v[i]) : v[i], E.up, E.last, E.n_bins, b[i])
                           : -1;
    }
}

struct DmumuLaunch {
    const void* mu;            // element (p, s) at mu[p * sp + s * ss], Float32 or Float64
    int64_t sp, ss;
    int64_t n, nsave;
    const int64_t* lags;       // this batch's lags
    int nl;                    // lags in this batch
    const double* edges;
    int n_bins, bin_abs;
    int ppc, groups, parts;    // particle slots per CTA, 8 * NS-lag groups, warps sharing a (slot, group)
    int slot_bytes;            // shared memory of a slot
    char* gslots;              // global staging of the slots' series and lists, when they do not fit on chip
    size_t gslot_bytes;
    // per-CTA outputs
    unsigned long long* part_cnt;  // [grid][n_bins][nl]
    double* part_sd;
    double* part_sd2;
    WelfordPart* part_w;           // [grid][nl]
};

// Where a slot's series lives: on chip with every value stored kStartLanes
// times (REP), on chip once (COMPACT), or in global memory (GLOBAL).
//
// REP: value s occupies 16 bytes (4 floats or 2 doubles), and start lane j reads
// its own copy.  The bank of lane (j, l) is then 4 ((s_j + L_l) mod 8) + j:
// the 32 reads of a row are conflict-free, whatever the four starts, when the
// set's lags differ mod 8, and the lags are dealt to the sets by their residue.
// With one copy the banks of 4 unrelated starts collide 3 to 4 ways.
enum { SLOT_REP = 0, SLOT_COMPACT = 1, SLOT_GLOBAL = 2 };

__host__ __device__ constexpr size_t up16(size_t v) { return (v + 15) & ~(size_t)15; }
// address units of one save: bytes on chip, values in global memory
__host__ __device__ constexpr int slot_stride(int mode, int mu_bytes)
{
    return mode == SLOT_REP ? 16 : (mode == SLOT_COMPACT ? mu_bytes : 1);
}
// added to an address, or in its place: past every valid one, and twice it does not wrap
constexpr unsigned kFar = 0x7fffffffu;

// shared memory of the CTA ahead of the slots
struct DmumuFixed {
    size_t edges, lag, sorted, rank, lane, total;  // hist2 comes first
};
__host__ __device__ inline DmumuFixed dmumu_fixed(int nl, int n_bins, int mu_bytes, int lanes, int ktab)
{
    DmumuFixed f;
    f.edges = up16(sizeof(unsigned) * (size_t)n_bins * (nl + 1));
    f.lag = up16(f.edges + (size_t)mu_bytes * (n_bins + 1));
    f.sorted = f.lag + sizeof(int) * nl;
    f.rank = f.sorted + sizeof(int) * nl;
    f.lane = f.rank + sizeof(int) * nl;
    f.total = up16(up16(f.lane + sizeof(int) * lanes) + ktab);
    return f;
}
// shared memory of a slot: series | list | hist[2][B] | cur[B + 1], next[B] |
// welford[nl] | tot_sd2[nl] | tot_c[nl] | nfin, with B = 2 (nb + 1) buckets
// (series and list elsewhere when GLOBAL)
struct DmumuSlot {
    size_t list, hist, cur, welford, tot, totc, nfin, total;
};
__host__ __device__ inline DmumuSlot dmumu_slot(int mode, int64_t nsave, int mu_bytes, int nl, int n_bins)
{
    DmumuSlot o;
    o.list = mode == SLOT_GLOBAL ? 0 : up16((size_t)nsave * slot_stride(mode, mu_bytes));
    o.hist = mode == SLOT_GLOBAL ? 0 : o.list + up16((size_t)nsave * 2);
    o.cur = o.hist + sizeof(int) * 4 * (n_bins + 1);
    o.welford = up16(o.cur + sizeof(int) * (4 * (n_bins + 1) + 1));
    o.tot = o.welford + sizeof(WelfordPart) * nl;
    o.totc = o.tot + sizeof(double) * nl;
    o.nfin = o.totc + sizeof(int) * nl;
    o.total = up16(o.nfin + sizeof(int));
    return o;
}

// Shared-memory load at a 32-bit window address: the pair loop then has one
// integer add per pair.  Not volatile, so that the loads of a row can overlap;
// every address comes from the start list, which is read after the barrier that
// publishes the series.
template <typename MuT>
__device__ __forceinline__ MuT lds(unsigned at)
{
    MuT v;
    if constexpr (sizeof(MuT) == 4) asm("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(at));
    else asm("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(at));
    return v;
}

__device__ __forceinline__ void slot_barrier(int slot, int threads)
{
    asm volatile("bar.sync %0, %1;" ::"r"(slot + 1), "r"(threads) : "memory");
}

template <typename MuT>
__device__ __forceinline__ void put_rep(void* series, int s, MuT v)
{
    if constexpr (sizeof(MuT) == 4) ((float4*)series)[s] = make_float4(v, v, v, v);
    else ((double2*)series)[s] = make_double2(v, v);
}

// A lag set whose lags reach past the end of the series from few starts only
// needs no test for most of them: the last kLongSets sets hold the longest lags,
// the others the rest, and a start is "clear" when even the longest of the
// others stays inside the series.
__host__ __device__ constexpr int long_sets(int ns) { return ns >= 6 ? 2 : 1; }

// v[q0 + j] summed over the four start lanes, on start lane j (0 beyond NS).
template <int NS, typename T>
__device__ __forceinline__ T start_sum(const T (&v)[NS], int q0, int j)
{
    const T z = T(0);
    const T v0 = q0 < NS ? v[q0 < NS ? q0 : 0] : z, v1 = q0 + 1 < NS ? v[q0 + 1 < NS ? q0 + 1 : 0] : z,
            v2 = q0 + 2 < NS ? v[q0 + 2 < NS ? q0 + 2 : 0] : z, v3 = q0 + 3 < NS ? v[q0 + 3 < NS ? q0 + 3 : 0] : z;
    const bool hi = j & 2, odd = j & 1;
    const T a = (hi ? v2 : v0) + __shfl_xor_sync(0xffffffffu, hi ? v0 : v2, 2 * kLagLanes);
    const T b = (hi ? v3 : v1) + __shfl_xor_sync(0xffffffffu, hi ? v1 : v3, 2 * kLagLanes);
    return (odd ? b : a) + __shfl_xor_sync(0xffffffffu, odd ? a : b, kLagLanes);
}

// Saves and list positions in loops that run up to some blocks past the end: unsigned
// where a series may hold nearly 2^31 saves, in global memory; at most 65,535 are on
// chip.
template <int MODE>
using SavePos = std::conditional_t<MODE == SLOT_GLOBAL, unsigned, int>;

// Pairs of one slot's share [r0, r1) of the start list, r0 in bin b.  The buckets of the list are
// (bin, clear starts), (bin, other starts) for every bin.  TEST: the series has NaN
// between finite saves, so the partner is tested and the pairs counted.
//
// A pair that does not exist reads the start itself and adds (+0, 0): a select
// on the address.  Predicates on the pair's arithmetic cost more (they become
// two selects for each double).
template <typename MuT, typename IdxT, int NS, int MODE, bool TEST>
__device__ __forceinline__ void dmumu_pairs(const MuT* series,
                                            const IdxT* list, const int* cur, bool clear_ok, int nb, int nl, int b,
                                            SavePos<MODE> r0, SavePos<MODE> r1, int end_save,
                                            const unsigned (&off)[NS], int lane,
                                            const int* lane_lag, double* out_sd, double* out_sd2,
                                            unsigned long long* out_cnt, double* tot_sd2, int* tot_c)
{
    using Pos = SavePos<MODE>;
    constexpr unsigned kStride = slot_stride(MODE, sizeof(MuT));
    constexpr int kOwn = (NS + kStartLanes - 1) / kStartLanes, kShort = NS - long_sets(NS);
    const int j = lane / kLagLanes, l = lane % kLagLanes;
    const unsigned copy = MODE == SLOT_REP ? (unsigned)(j % (16 / (int)sizeof(MuT))) * (unsigned)sizeof(MuT) : 0u;
    const unsigned base = (MODE == SLOT_GLOBAL ? 0u : (unsigned)__cvta_generic_to_shared(series)) + copy;
    const unsigned end = base - copy + (unsigned)end_save * kStride;
    auto value = [&](unsigned at) -> MuT {
        if constexpr (MODE == SLOT_GLOBAL) return series[at];
        else return lds<MuT>(at);
    };
    int mine[kOwn];  // the lags whose sums this lane flushes
#pragma unroll
    for (int q = 0; q < kOwn; ++q) mine[q] = 4 * q + j < NS ? lane_lag[(4 * q + j) * kLagLanes + l] : -1;
    double own[kOwn];
    int ownc[TEST ? kOwn : 1];
#pragma unroll
    for (int k = 0; k < kOwn; ++k) own[k] = 0.0;
#pragma unroll
    for (int k = 0; k < (TEST ? kOwn : 1); ++k) ownc[k] = 0;
    for (Pos e = r0; e < r1; ++b) {
        const Pos e1 = min((Pos)cur[2 * b + 2], r1);
        if (e >= e1) continue;
        double sd[NS], sq[NS];
        int c[TEST ? NS : 1];
#pragma unroll
        for (int k = 0; k < NS; ++k) sd[k] = sq[k] = 0.0;
#pragma unroll
        for (int k = 0; k < (TEST ? NS : 1); ++k) c[k] = 0;
        if constexpr (!TEST && MODE != SLOT_GLOBAL) {
            // whole rows of clear starts
            const Pos ec = clear_ok ? e + ((min((Pos)cur[2 * b + 1], e1) - e) & ~(kStartLanes - 1)) : e;
#pragma unroll 2
            for (; e < ec; e += kStartLanes) {
                const unsigned at = base + list[e + j] * kStride;
                const double a = (double)value(at);
#pragma unroll
                for (int k = 0; k < NS; ++k) {
                    unsigned addr = at + off[k];
                    if (k >= kShort) addr = addr < end ? addr : at;
                    const double d = (double)value(addr) - a;
                    sd[k] += d;
                    sq[k] = fma(d, d, sq[k]);
                }
            }
        }
        for (; e < e1; e += kStartLanes) {
            const unsigned at = base + list[min(e + j, e1 - 1)] * kStride;
            const double a = (double)value(at);
            const unsigned from = e + j < e1 ? at : kFar;
#pragma unroll
            for (int k = 0; k < NS; ++k) {
                const unsigned addr = from + off[k];
                const MuT w = value(addr < end ? addr : at);
                if constexpr (TEST) {
                    const bool ok = addr < end && w == w;
                    const double d = ok ? (double)w - a : 0.0;
                    sd[k] += d;
                    sq[k] = fma(d, d, sq[k]);
                    c[k] += ok;
                } else {
                    const double d = (double)w - a;
                    sd[k] += d;
                    sq[k] = fma(d, d, sq[k]);
                }
            }
        }
        // the four starts' sums of set 4 q + j end up on the start lane j, which
        // flushes them: whole warps per flush, not one set's 8 lanes at a time
#pragma unroll
        for (int q = 0; q < kOwn; ++q) {
            const double fd = start_sum<NS>(sd, 4 * q, j), fq = start_sum<NS>(sq, 4 * q, j);
            own[q] += fq;
            int fc = 0;
            if constexpr (TEST) {
                fc = start_sum<NS>(c, 4 * q, j);
                ownc[q] += fc;
            }
            if (b < nb && mine[q] >= 0) {
                // straight to the CTA's partials in L2: reductions that nothing
                // waits for (a shared-memory double add is a compare-and-swap
                // loop: 2,200 cycles a flush)
                const int ai = b * nl + mine[q];  // [bin][lag]
                atomicAdd(&out_sd[ai], fd);
                atomicAdd(&out_sd2[ai], fq);
                if constexpr (TEST)
                    if (fc > 0) atomicAdd(&out_cnt[ai], (unsigned long long)fc);
            }
        }
        e = e1;
    }
#pragma unroll
    for (int q = 0; q < kOwn; ++q) {
        if (mine[q] < 0) continue;
        if (own[q] != 0.0) atomicAdd(&tot_sd2[mine[q]], own[q]);
        if constexpr (TEST)
            if (ownc[q] > 0) atomicAdd(&tot_c[mine[q]], ownc[q]);
    }
}

template <typename MuT, int NS, int MODE>
__global__ void __launch_bounds__(max_threads(NS), 1) dmumu_kernel(DmumuLaunch a)
{
    using IdxT = std::conditional_t<MODE == SLOT_GLOBAL, uint32_t, uint16_t>;
    extern __shared__ __align__(16) unsigned char smem[];
    const int nb = a.n_bins, nl = a.nl, nsave = (int)a.nsave;
    const int sets = a.groups * NS;
    const int ktab_bytes = MODE == SLOT_REP ? nsave + 1 : 0;
    const DmumuFixed F = dmumu_fixed(nl, nb, sizeof(MuT), sets * kLagLanes, ktab_bytes);
    unsigned* hist2 = (unsigned*)smem;  // [bin][k]: starts that reach k lags
    MuT* s_edge = (MuT*)(smem + F.edges);
    int* s_lag = (int*)(smem + F.lag);        // lag in saves, nsave when no pair exists
    int* s_sorted = (int*)(smem + F.sorted);  // ascending
    int* s_rank = (int*)(smem + F.rank);      // position of each lag in s_sorted
    int* s_lane = (int*)(smem + F.lane);      // lag of (set, lag lane), -1: idle
    uint8_t* ktab = smem + up16(F.lane + sizeof(int) * (size_t)sets * kLagLanes);  // [x]: lags below x (REP)
    const int64_t cta = blockIdx.x;
    unsigned long long* out_cnt = a.part_cnt + cta * nl * nb;  // [bin][lag]
    double* out_sd = a.part_sd + cta * nl * nb;
    double* out_sd2 = a.part_sd2 + cta * nl * nb;

    for (int i = threadIdx.x; i < nl * nb; i += blockDim.x) {
        out_cnt[i] = 0ull;
        out_sd[i] = 0.0;
        out_sd2[i] = 0.0;
    }
    __threadfence();
    for (int i = threadIdx.x; i < nb * (nl + 1); i += blockDim.x) hist2[i] = 0u;
    for (int i = threadIdx.x; i <= nb; i += blockDim.x) s_edge[i] = edge_up(a.edges[i], MuT());
    for (int i = threadIdx.x; i < sets * kLagLanes; i += blockDim.x) s_lane[i] = -1;
    for (int i = threadIdx.x; i < nl; i += blockDim.x) {
        const int64_t L = a.lags[i];
        s_lag[i] = (L < 1 || L >= a.nsave) ? nsave : (int)L;  // reference: lag >= nsteps -> skipped
    }
    const double span = a.edges[nb] - a.edges[0];
    BinEdges<MuT> E{s_edge, edge_up(a.edges[0], MuT()), edge_down(a.edges[nb], MuT()),
                    span > 0.0 && isfinite(span) ? (MuT)((double)nb / span) : MuT(0), nb, a.bin_abs};
    if (!isfinite(E.inv_w)) E.inv_w = MuT(0);
    __syncthreads();
    // lags by value; then dealt to the short and to the long sets, each in the
    // order of their residue mod 8 so that the lags of a set differ in it where
    // possible
    for (int i = threadIdx.x; i < nl; i += blockDim.x) {
        const int L = s_lag[i];
        int rank = 0;
        for (int q = 0; q < nl; ++q) rank += s_lag[q] < L || (s_lag[q] == L && q < i);
        s_rank[i] = rank;
        s_sorted[rank] = L;
    }
    __syncthreads();
    const int n_long = a.groups * long_sets(NS), n_short = sets - n_long;
    const int short_lags = min(nl, n_short * kLagLanes);
    for (int i = threadIdx.x; i < nl; i += blockDim.x) {
        const int r = s_lag[i] % kLagLanes;
        const bool is_short = s_rank[i] < short_lags;
        int pos = 0;
        for (int q = 0; q < nl; ++q) {
            const int rq = s_lag[q] % kLagLanes;
            pos += (s_rank[q] < short_lags) == is_short && (rq < r || (rq == r && q < i));
        }
        // set k of group g is at g * NS + k, the long ones last
        const int pool = is_short ? n_short : n_long, set = pos % pool, per = pool / a.groups;
        s_lane[((set / per) * NS + (is_short ? 0 : NS - long_sets(NS)) + set % per) * kLagLanes + pos / pool] = i;
    }
    __syncthreads();
    // starts below this reach every lag of the short sets (in a whole series)
    const int clear_end = short_lags > 0 ? max(0, nsave - s_sorted[short_lags - 1]) : nsave;
    auto lags_below = [&](int x) {
        int k = 0;
        for (int hi = nl; k < hi;) {
            const int m = (k + hi) >> 1;
            if (s_sorted[m] < x) k = m + 1;
            else hi = m;
        }
        return k;
    };
    if constexpr (MODE == SLOT_REP)
        for (int x = threadIdx.x; x <= nsave; x += blockDim.x) ktab[x] = (uint8_t)lags_below(x);

    const int warp = threadIdx.x / kWarp, lane = threadIdx.x % kWarp;
    const int wps = a.groups * a.parts;  // warps per particle slot
    const int slot = warp / wps, wis = warp % wps;
    const int group = wis % a.groups, part = wis / a.groups;
    const int st = wis * kWarp + lane, T = wps * kWarp;  // thread within the slot
    unsigned char* sb = smem + F.total + (size_t)slot * a.slot_bytes;
    const DmumuSlot O = dmumu_slot(MODE, a.nsave, sizeof(MuT), nl, nb);
    char* gb = MODE == SLOT_GLOBAL ? a.gslots + (cta * a.ppc + slot) * a.gslot_bytes : nullptr;
    MuT* series = MODE == SLOT_GLOBAL ? (MuT*)gb : (MuT*)sb;
    IdxT* list = MODE == SLOT_GLOBAL ? (IdxT*)(gb + up16(sizeof(MuT) * (size_t)a.nsave)) : (IdxT*)(sb + O.list);
    // buckets of the start list: 2 b + (0: clear, 1: not) of bin b
    const int nbk = 2 * (nb + 1);
    int* hist = (int*)(sb + O.hist);     // starts per bucket whose rank a thread keeps, then the others
    int* hist_r = hist + nbk;
    int* cur = (int*)(sb + O.cur);       // first list entry of each bucket; cur[nbk] = all
    int* next = cur + nbk + 1;           // next free entry for a start whose rank was not kept
    WelfordPart* wel = (WelfordPart*)(sb + O.welford);
    double* tot_sd2 = (double*)(sb + O.tot);
    int* tot_c = (int*)(sb + O.totc);
    int* nfin_s = (int*)(sb + O.nfin);
    for (int i = st; i < 2 * nbk; i += T) hist[i] = 0;
    for (int i = st; i < nl; i += T) {
        wel[i] = WelfordPart{0, 0.0, 0.0, 0.0, 0};
        tot_sd2[i] = 0.0;
        tot_c[i] = 0;
    }
    if (st == 0) *nfin_s = nsave;
    __syncthreads();

    unsigned off[NS];
#pragma unroll
    for (int k = 0; k < NS; ++k) {
        const int li = s_lane[(group * NS + k) * kLagLanes + lane % kLagLanes];
        const int L = li >= 0 ? s_lag[li] : 0;  // an idle lane pairs a start with itself
        off[k] = L < nsave ? (unsigned)L * (unsigned)slot_stride(MODE, sizeof(MuT)) : kFar;
    }
    const MuT* mu = (const MuT*)a.mu;
    const int64_t step = (int64_t)gridDim.x * a.ppc, hop = T * a.ss;
    using Pos = SavePos<MODE>;
    const Pos n_saves = (Pos)nsave, clear_from = (Pos)clear_end;
    for (int64_t p = cta * a.ppc + slot; p < a.n; p += step) {
        const MuT* row = mu + p * a.sp + st * a.ss;
        // ---- stage the series and count the starts per bucket, kBatch saves of a
        // thread side by side (one after another they are a chain of a load, a
        // conversion, two shared reads and an atomic each)
        uint32_t pk[kKeep];  // bucket << 16 | rank within it, ~0: not a start
        {
            int bad = nsave;
            const MuT* q = row;
            auto stage = [&](Pos s0, int (&b)[kBatch]) {
                MuT v[kBatch];
#pragma unroll
                for (int i = 0; i < kBatch; ++i) v[i] = s0 + i * T < n_saves ? q[i * hop] : MuT(NAN);
                bins_of(v, E, b);
#pragma unroll
                for (int i = 0; i < kBatch; ++i) {
                    const Pos s = s0 + i * T;
                    if (s < n_saves) {
                        const MuT x = b[i] >= 0 ? v[i] : MuT(NAN);
                        if constexpr (MODE == SLOT_REP) put_rep(series, s, x);
                        else series[s] = x;
                        if (b[i] < 0) bad = min(bad, (int)s);
                    }
                }
                q += kBatch * hop;
            };
#pragma unroll
            for (int i0 = 0; i0 < kKeep; i0 += kBatch) {
                if (i0 * T >= nsave) break;
                int b[kBatch];
                stage(i0 * T + st, b);
#pragma unroll
                for (int i = 0; i < kBatch; ++i) {
                    const int k = 2 * b[i] + ((i0 + i) * T + st >= clear_end);
                    pk[i0 + i] = b[i] < 0 ? 0xffffffffu : (uint32_t)k << 16 | (uint32_t)atomicAdd(&hist[k], 1);
                }
            }
            for (Pos s0 = kKeep * T + st; s0 < n_saves; s0 += kBatch * T) {
                int b[kBatch];
                stage(s0, b);
#pragma unroll
                for (int i = 0; i < kBatch; ++i)
                    if (b[i] >= 0) atomicAdd(&hist_r[2 * b[i] + (s0 + i * T >= clear_from)], 1);
            }
            if (bad < nsave) atomicMin(nfin_s, bad);
        }
        slot_barrier(slot, T);
        // ---- first list entry of each bucket: a lane adds a run of them
        if (wis == 0) {
            const int per = (nbk + kWarp - 1) / kWarp, b0 = min(lane * per, nbk), b1 = min(b0 + per, nbk);
            int t = 0;
            for (int b = b0; b < b1; ++b) t += hist[b] + hist_r[b];
            int incl = t;
#pragma unroll
            for (int d = 1; d < kWarp; d <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, incl, d);
                if (lane >= d) incl += y;
            }
            int run = incl - t;
            for (int b = b0; b < b1; ++b) {
                const int h = hist[b];
                cur[b] = run;
                next[b] = run + h;
                run += h + hist_r[b];
            }
            if (lane == kWarp - 1) cur[nbk] = run;
        }
        slot_barrier(slot, T);
        const int nfin = *nfin_s, total = cur[nbk];
        const bool prefix = total == nfin;  // every finite save comes before the first non-finite one
        // ---- the list, and the lags each start reaches (beyond kKeep saves per
        // thread the bin is computed again)
        {
            auto reach = [&](int s, int b) {
                if (!prefix || b >= nb) return;
                const int k = MODE == SLOT_REP ? (int)ktab[nfin - s] : lags_below(nfin - s);
                atomicAdd(&hist2[b * (nl + 1) + k], 1u);
            };
#pragma unroll
            for (int i = 0; i < kKeep; ++i) {
                if (i * T >= nsave) break;
                if (pk[i] == 0xffffffffu || i * T + st >= nsave) continue;
                const int k = (int)(pk[i] >> 16);
                list[cur[k] + (int)(pk[i] & 0xffffu)] = (IdxT)(i * T + st);
                reach(i * T + st, k >> 1);
            }
            for (Pos s0 = kKeep * T + st; s0 < n_saves; s0 += kBatch * T) {
                MuT v[kBatch];
                int b[kBatch], at[kBatch];
#pragma unroll
                for (int i = 0; i < kBatch; ++i) {
                    const Pos s = s0 + i * T;
                    if constexpr (MODE == SLOT_REP)
                        v[i] = s < n_saves ? *(const MuT*)((const char*)series + 16 * (size_t)s) : MuT(NAN);
                    else
                        v[i] = s < n_saves ? series[s] : MuT(NAN);
                }
                bins_of(v, E, b);
#pragma unroll
                for (int i = 0; i < kBatch; ++i)
                    at[i] = b[i] >= 0 ? atomicAdd(&next[2 * b[i] + (s0 + i * T >= clear_from)], 1) : 0;
#pragma unroll
                for (int i = 0; i < kBatch; ++i) {
                    if (b[i] < 0) continue;
                    list[at[i]] = (IdxT)(s0 + i * T);
                    reach((int)(s0 + i * T), b[i]);
                }
            }
        }
        slot_barrier(slot, T);
        for (int i = st; i < 2 * nbk; i += T) hist[i] = 0;
        if (st == 0) *nfin_s = nsave;
        // ---- pairs: shares of the list of equal cost, a flush counted as
        // kFlushCost starts (a bin may straddle two shares; each flushes its
        // part of it)
        int bin0 = 0, bin1 = 0;
        auto boundary = [&](int k, int& b) {
            const Pos all = (Pos)total + kFlushCost * (nb + 1);  // in 32 bits either way
            const Pos target = (Pos)(((unsigned long long)all * k) / a.parts);
            b = 0;
            for (int hi = nb + 1; b + 1 < hi;) {
                const int m = (b + hi) >> 1;
                if ((Pos)cur[2 * m] + kFlushCost * m <= target) b = m;
                else hi = m;
            }
            // the flushes up to b come before target: the chosen m passed that test
            return min((Pos)cur[2 * b + 2], max((Pos)cur[2 * b], target - kFlushCost * b));
        };
        const Pos r0 = boundary(part, bin0), r1 = part + 1 == a.parts ? (Pos)total : boundary(part + 1, bin1);
        const int* lane_lag = s_lane + group * NS * kLagLanes;
        if (prefix)
            dmumu_pairs<MuT, IdxT, NS, MODE, false>(series, list, cur, nfin == nsave, nb, nl, bin0, r0, r1,
                                                    nfin, off, lane, lane_lag, out_sd, out_sd2, out_cnt, tot_sd2,
                                                    tot_c);
        else
            dmumu_pairs<MuT, IdxT, NS, MODE, true>(series, list, cur, false, nb, nl, bin0, r0, r1, nsave,
                                                   off, lane, lane_lag, out_sd, out_sd2, out_cnt, tot_sd2, tot_c);
        slot_barrier(slot, T);
        // ---- per-particle value: mean dmu^2 over its valid pairs (dmumu:528-537).
        // The next particle's staging may start: what it shares with this (hist,
        // nfin) was reset after its last read, before the barrier above, and
        // tot_* are next added to three barriers on.
        for (int i = st; i < nl; i += T) {
            const int tc = prefix ? max(0, nfin - s_lag[i]) : tot_c[i];
            const double ts = tot_sd2[i];
            if (tc > 0) {
                WelfordPart w = wel[i];
                const double value = ts / (double)tc;
                w.count += 1;
                const double delta = value - w.mean;
                w.mean += delta / (double)w.count;
                w.m2 += delta * (value - w.mean);
                w.pair_ss += ts;
                w.pair_n += tc;
                wel[i] = w;
            }
            tot_sd2[i] = 0.0;
            tot_c[i] = 0;
        }
    }

    // ---- CTA epilogue: (bin, lag) sums and counts, Welford triples in slot order
    __syncthreads();
    for (int b = threadIdx.x; b < nb; b += blockDim.x) {
        unsigned run = 0;
        for (int k = nl; k >= 0; --k) {
            run += hist2[b * (nl + 1) + k];
            hist2[b * (nl + 1) + k] = run;
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < nl * nb; i += blockDim.x) {
        const unsigned c = hist2[i / nl * (nl + 1) + s_rank[i % nl] + 1];  // starts that reach more lags than this one's rank
        if (c) atomicAdd(&out_cnt[i], (unsigned long long)c);
    }
    for (int l = threadIdx.x; l < nl; l += blockDim.x) {
        WelfordPart r{0, 0.0, 0.0, 0.0, 0};
        for (int sl = 0; sl < a.ppc; ++sl) {
            const WelfordPart q = ((const WelfordPart*)(smem + F.total + (size_t)sl * a.slot_bytes + O.welford))[l];
            welford_merge(r.count, r.mean, r.m2, q.count, q.mean, q.m2);
            r.pair_ss += q.pair_ss;
            r.pair_n += q.pair_n;
        }
        a.part_w[cta * nl + l] = r;
    }
}

// Reduce per-CTA partials and add / merge into the outputs.  Blocks below
// `cells` take 32 (lag, bin) cells each: 32 threads per cell add the CTAs
// g = y, y + 32, ... and the 32 sums are added in order.  Each further block
// merges one lag's Welford triples: thread t takes the CTAs t, t + 1024, ..., then
// a tree over the threads.  Both orders are fixed.  The kernel is a chain of
// L2 reads and FP64 divisions, so it runs as wide as the partials allow: one
// thread per cell walking all CTAs took 130 us for any size, half of a
// 4096-particle call.
constexpr int kFinRows = 32;
__global__ void __launch_bounds__(kWarp* kFinRows)
    dmumu_finalize_kernel(const unsigned long long* __restrict__ part_cnt, const double* __restrict__ part_sd,
                          const double* __restrict__ part_sd2, const WelfordPart* __restrict__ part_w, int grid, int nl,
                          int nb, int lag0, int cells, int64_t* counts, double* sum_d, double* sum_d2,
                          int64_t* w_count, double* w_mean, double* w_m2, double* pair_ss, int64_t* pair_n)
{
    const int x = threadIdx.x % kWarp, y = threadIdx.x / kWarp;
    if ((int)blockIdx.x < cells) {
        __shared__ unsigned long long sc[kFinRows][kWarp];
        __shared__ double ss[kFinRows][kWarp], ss2[kFinRows][kWarp];
        const int t = blockIdx.x * kWarp + x;
        unsigned long long c = 0;
        double sd = 0.0, sd2 = 0.0;
        if (t < nl * nb) {
#pragma unroll 4
            for (int g = y; g < grid; g += kFinRows) {
                const int64_t q = (int64_t)g * nl * nb + t;
                c += part_cnt[q];
                sd += part_sd[q];
                sd2 += part_sd2[q];
            }
        }
        sc[y][x] = c;
        ss[y][x] = sd;
        ss2[y][x] = sd2;
        __syncthreads();
        if (y == 0 && t < nl * nb) {
#pragma unroll
            for (int r = 1; r < kFinRows; ++r) {
                c += sc[r][x];
                sd += ss[r][x];
                sd2 += ss2[r][x];
            }
            const int l = t % nl, b = t / nl;                // partials are [bin][lag]
            const int64_t o = (int64_t)(lag0 + l) * nb + b;  // Julia (n_bins, n_lags)
            counts[o] += (int64_t)c;
            sum_d[o] += sd;
            sum_d2[o] += sd2;
        }
        return;
    }
    __shared__ WelfordPart sw[kWarp];
    const int t = (int)blockIdx.x - cells;
    WelfordPart r{0, 0.0, 0.0, 0.0, 0};
    auto merge = [&](const WelfordPart& q) {
        welford_merge(r.count, r.mean, r.m2, q.count, q.mean, q.m2);
        r.pair_ss += q.pair_ss;
        r.pair_n += q.pair_n;
    };
    auto tree = [&]() {  // over a warp, into lane 0
#pragma unroll
        for (int o = kWarp / 2; o > 0; o >>= 1)
            merge(WelfordPart{__shfl_down_sync(0xffffffffu, r.count, o), __shfl_down_sync(0xffffffffu, r.mean, o),
                              __shfl_down_sync(0xffffffffu, r.m2, o), __shfl_down_sync(0xffffffffu, r.pair_ss, o),
                              __shfl_down_sync(0xffffffffu, r.pair_n, o)});
    };
    for (int g = threadIdx.x; g < grid; g += blockDim.x) merge(part_w[(int64_t)g * nl + t]);
    if (y * kWarp < grid) tree();
    if (x == 0) sw[y] = r;
    __syncthreads();
    if (y != 0) return;
    r = sw[x];
    tree();
    if (x == 0) {
        const int l = lag0 + t;
        long long gc = w_count[l];
        double gm = w_mean[l], gm2 = w_m2[l];
        welford_merge(gc, gm, gm2, r.count, r.mean, r.m2);
        w_count[l] = gc;
        w_mean[l] = gm;
        w_m2[l] = gm2;
        pair_ss[l] += r.pair_ss;
        pair_n[l] += r.pair_n;
    }
}

// Injection estimator (dmumu:562-654): one start, save 0, per particle.  A CTA
// takes tiles of particles: saves 0 and the lags' are staged in shared memory --
// along the particles when those are the near ones in memory, along the lags
// otherwise -- and a warp then walks particles with a lag per lane, so that the
// bin is the same for the whole warp and a flush hits consecutive words.  Sums
// stay in registers while the bin does not change (all particles of a fixed-mu
// injection start in one bin).  The particles' dmu^2 enter the lag's Welford
// triple a tile at a time, as shifted sums about the running mean.
//
// It moves the (lags + 1) saves that the estimator needs instead of the whole
// series.
constexpr int kInjThreads = 512;

struct DmumuInjection {
    const void* mu;            // element (p, s) at mu[p * sp + s * ss]
    int64_t sp, ss;
    int packed;                // 1: the series holds save 0 and then lag saves, this batch's from `first` on
    int first;
    int64_t n, nsave;
    const int64_t* lags;
    int nl;
    const double* edges;
    int n_bins, bin_abs;
    int tile;                  // particles per tile
    unsigned long long* part_cnt;
    double* part_sd;
    double* part_sd2;
    WelfordPart* part_w;
};

struct DmumuInjFixed {
    size_t sd2, cnt, edges, at, bin, wel, tile, total;
};
__host__ __device__ inline DmumuInjFixed dmumu_inj_fixed(int nl, int n_bins, int mu_bytes, int tile)
{
    DmumuInjFixed f;
    f.sd2 = (size_t)nl * n_bins * sizeof(double);
    f.cnt = 2 * f.sd2;
    f.edges = up16(f.cnt + sizeof(unsigned) * (size_t)nl * n_bins);
    f.at = up16(f.edges + (size_t)mu_bytes * (n_bins + 1));
    f.bin = f.at + sizeof(int64_t) * (nl + 1);
    f.tile = up16(f.bin + sizeof(int) * tile);
    f.wel = f.tile;  // the warps' Welford triples take the tile's place at the end
    const size_t t = (size_t)mu_bytes * (nl + 1) * (tile + 1), w = sizeof(WelfordPart) * kInjThreads;
    f.total = f.tile + up16(t > w ? t : w);
    return f;
}

template <typename MuT>
__global__ void __launch_bounds__(kInjThreads) dmumu_injection_kernel(DmumuInjection a)
{
    extern __shared__ __align__(16) unsigned char smem[];
    const int nb = a.n_bins, nl = a.nl, P = a.tile, rows = nl + 1;
    const DmumuInjFixed F = dmumu_inj_fixed(nl, nb, sizeof(MuT), P);
    double* acc_sd = (double*)smem;  // [bin][lag]
    double* acc_sd2 = (double*)(smem + F.sd2);
    unsigned* acc_cnt = (unsigned*)(smem + F.cnt);
    MuT* s_edge = (MuT*)(smem + F.edges);
    int64_t* s_at = (int64_t*)(smem + F.at);  // element offset of each staged save, -1: no such save
    int* s_bin = (int*)(smem + F.bin);
    MuT* tile = (MuT*)(smem + F.tile);        // [save][particle], padded by one
    for (int i = threadIdx.x; i < nl * nb; i += blockDim.x) {
        acc_sd[i] = 0.0;
        acc_sd2[i] = 0.0;
        acc_cnt[i] = 0u;
    }
    for (int i = threadIdx.x; i <= nb; i += blockDim.x) s_edge[i] = edge_up(a.edges[i], MuT());
    for (int i = threadIdx.x; i < rows; i += blockDim.x) {
        const int64_t L = i == 0 ? 0 : a.lags[i - 1];
        const bool ok = i == 0 || (L >= 1 && L < a.nsave);  // reference: lag >= nsteps -> skipped
        s_at[i] = !ok ? -1 : (a.packed && i > 0 ? (int64_t)(a.first + i - 1) : L) * a.ss;
    }
    const double span = a.edges[nb] - a.edges[0];
    BinEdges<MuT> E{s_edge, edge_up(a.edges[0], MuT()), edge_down(a.edges[nb], MuT()),
                    span > 0.0 && isfinite(span) ? (MuT)((double)nb / span) : MuT(0), nb, a.bin_abs};
    if (!isfinite(E.inv_w)) E.inv_w = MuT(0);
    const int warp = threadIdx.x / kWarp, lane = threadIdx.x % kWarp, warps = kInjThreads / kWarp;
    const int groups = (nl + kWarp - 1) / kWarp;  // at most 8 of the 16 warps
    const int subs = warps / groups, group = warp % groups, sub = warp / groups;
    const int li = group * kWarp + lane;
    const bool on = sub < subs && li < nl;
    const MuT* mu = (const MuT*)a.mu;
    const bool particles_near = a.sp <= a.ss;
    long long wc = 0, pn = 0;
    double wm = 0.0, wm2 = 0.0, pss = 0.0;
    int bin = -1;
    unsigned c = 0;
    double sd = 0.0, sq = 0.0;
    auto flush = [&]() {
        if (bin >= 0 && bin < nb && on && c > 0) {
            const int ai = bin * nl + li;
            atomicAdd(&acc_cnt[ai], c);
            atomicAdd(&acc_sd[ai], sd);
            atomicAdd(&acc_sd2[ai], sq);
        }
        c = 0;
        sd = sq = 0.0;
    };
    __syncthreads();
    for (int64_t p0 = (int64_t)blockIdx.x * P; p0 < a.n; p0 += (int64_t)gridDim.x * P) {
        const int np = (int)min((int64_t)P, a.n - p0);
        if (particles_near) {
            for (int r = warp; r < rows; r += warps) {
                const int64_t at = s_at[r];
                const MuT* src = mu + p0 * a.sp + (at >= 0 ? at : 0);
                MuT* dst = tile + r * (P + 1);
#pragma unroll 4
                for (int q = lane; q < np; q += kWarp) dst[q] = at >= 0 ? src[q * a.sp] : MuT(NAN);
            }
        } else {
            for (int q0 = warp; q0 < np; q0 += 4 * warps)
                for (int r = lane; r < rows; r += kWarp) {
                    const int64_t at = s_at[r];
                    MuT v[4];
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const int q = q0 + k * warps;
                        v[k] = at >= 0 && q < np ? mu[(p0 + q) * a.sp + at] : MuT(NAN);
                    }
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        if (q0 + k * warps < np) tile[r * (P + 1) + q0 + k * warps] = v[k];
                }
        }
        __syncthreads();
        for (int q = threadIdx.x; q < np; q += blockDim.x) {
            const MuT v[1] = {tile[q]};
            int b[1];
            bins_of(v, E, b);
            s_bin[q] = b[0];
        }
        __syncthreads();
        if (sub < subs) {
            const MuT* mine = tile + (1 + (on ? li : 0)) * (P + 1);
            int cn = 0;
            double s1 = 0.0, s2 = 0.0, shift = wm, ps = 0.0;
            for (int q = sub; q < np; q += subs) {
                const int b = s_bin[q];
                if (b < 0) continue;
                if (b != bin) {
                    flush();
                    bin = b;
                }
                const MuT w = mine[q];
                if (on && isfinite(w)) {
                    const double d = (double)w - (double)tile[q], v = d * d;
                    ++c;
                    sd += d;
                    sq += v;
                    if (wc == 0 && cn == 0) shift = v;
                    const double z = v - shift;
                    ++cn;
                    s1 += z;
                    s2 = fma(z, z, s2);
                    ps += v;
                }
            }
            if (cn > 0) {
                const double m = s1 / (double)cn;
                welford_merge(wc, wm, wm2, cn, shift + m, fmax(0.0, s2 - s1 * m));
                pss += ps;
                pn += cn;
            }
        }
        __syncthreads();
    }
    flush();
    WelfordPart* wp = (WelfordPart*)(smem + F.wel);
    wp[threadIdx.x] = WelfordPart{wc, wm, wm2, pss, pn};
    __syncthreads();
    const int64_t cta = blockIdx.x;
    for (int i = threadIdx.x; i < nl * nb; i += blockDim.x) {
        a.part_cnt[cta * nl * nb + i] = acc_cnt[i];
        a.part_sd[cta * nl * nb + i] = acc_sd[i];
        a.part_sd2[cta * nl * nb + i] = acc_sd2[i];
    }
    for (int l = threadIdx.x; l < nl; l += blockDim.x) {
        WelfordPart r{0, 0.0, 0.0, 0.0, 0};
        for (int s = 0; s < subs; ++s) {
            const WelfordPart q = wp[(s * groups + l / kWarp) * kWarp + l % kWarp];
            welford_merge(r.count, r.mean, r.m2, q.count, q.mean, q.m2);
            r.pair_ss += q.pair_ss;
            r.pair_n += q.pair_n;
        }
        a.part_w[cta * nl + l] = r;
    }
}

// ------------------------------------------------------------------ host side
// Limits of the call, the same for the allocating and the no-alloc entry.  The
// arithmetic (24 bytes per (lag, bin) cell, 200 KB) is the one that
// stats.dmumu_noalloc_fits and stats.dmumu_scratch_bound state for callers.
struct DmumuLimits {
    int nl_cap;          // lags per launch
    size_t fixed, slot;  // shared memory the bounds count for a CTA and for a series
};
constexpr size_t kDmumuBudget = 200 * 1024;

DmumuLimits dmumu_limits(const DmumuArgs& a, int mu_bytes)
{
    DmumuLimits m;
    m.nl_cap = (int)std::max<size_t>(32, ((kDmumuBudget / 2) / ((size_t)a.n_bins * 24)) / 32 * 32);
    m.nl_cap = std::min(m.nl_cap, 32 * 8);
    const int nl = std::min(m.nl_cap, a.n_lags);
    m.fixed = up16(sizeof(double) * (size_t)(a.n_bins + 1)) +
              std::max((size_t)nl * a.n_bins * 24, sizeof(WelfordPart) * (size_t)1024);
    m.slot = up16((size_t)(a.nsave + 1) * mu_bytes) + up16((size_t)a.nsave * (a.nsave <= 65535 ? 2 : 4)) +
             up16(sizeof(int) * (size_t)(8 * (a.n_bins + 1) + a.n_bins + 2)) + up16(16 * (size_t)m.nl_cap);
    return m;
}

// Launch shape of the sliding estimator for nl lags.
struct DmumuShape {
    int mode, ns, groups, parts, ppc;
    DmumuFixed fixed;
    DmumuSlot slot;
};

DmumuShape dmumu_shape(int64_t n, int64_t nsave, int nl, int n_bins, int mu_bytes, size_t max_smem, int num_sms)
{
    DmumuShape h{};
    const int sets = (nl + kLagLanes - 1) / kLagLanes;
    h.groups = (sets + kMaxSets - 1) / kMaxSets;
    auto set_mode = [&](int mode) {
        h.mode = mode;
        h.ns = (sets + h.groups - 1) / h.groups;
        // rounded up to an instance: a set without lags costs its share of the pair loop
        if (mode != SLOT_REP || mu_bytes == 8) h.ns = h.ns <= 4 ? 4 : 8;
        h.fixed = dmumu_fixed(nl, n_bins, mu_bytes, h.groups * h.ns * kLagLanes,
                              mode == SLOT_REP ? (int)nsave + 1 : 0);
        h.slot = dmumu_slot(mode, nsave, mu_bytes, nl, n_bins);
        return h.fixed.total + h.slot.total <= max_smem;
    };
    const bool short_index = nsave <= 65535;
    if (!(short_index && nl <= 255 && set_mode(SLOT_REP)) && !(short_index && set_mode(SLOT_COMPACT)))
        set_mode(SLOT_GLOBAL);
    int max_ppc = (int)std::min<size_t>(kMaxSlots, (max_smem - std::min(max_smem, h.fixed.total)) / h.slot.total);
    if (h.mode == SLOT_GLOBAL) max_ppc = std::min<int64_t>({max_ppc, 8, std::max<int64_t>(1, INT32_MAX / nsave)});
    max_ppc = (int)std::max<int64_t>(1, std::min<int64_t>(max_ppc, n));
    // rounds of particles times the time of one, which falls with the warps on
    // it but for a constant part (barriers, the scan); the larger ppc among equals
    double best = 0.0;
    for (int c = 1; c <= max_ppc && c * h.groups * kWarp <= max_threads(h.ns); ++c) {
        const int pt = std::max(1, max_threads(h.ns) / (kWarp * c * h.groups));
        const double rounds = (double)((n + (int64_t)c * num_sms - 1) / ((int64_t)c * num_sms));
        const double cost = rounds * (1.0 / pt + 0.02);
        if (best == 0.0 || cost <= best) {
            best = cost;
            h.ppc = c;
            h.parts = pt;
        }
    }
    return h;
}

template <typename MuT, int NS>
void* dmumu_fn_ns(int mode)
{
    return mode == SLOT_REP       ? (void*)dmumu_kernel<MuT, NS, SLOT_REP>
           : mode == SLOT_COMPACT ? (void*)dmumu_kernel<MuT, NS, SLOT_COMPACT>
                                  : (void*)dmumu_kernel<MuT, NS, SLOT_GLOBAL>;
}

template <typename MuT>
void* dmumu_fn(int mode, int ns)
{
    switch (ns) {
    case 1: return (void*)dmumu_kernel<float, 1, SLOT_REP>;
    case 2: return (void*)dmumu_kernel<float, 2, SLOT_REP>;
    case 3: return (void*)dmumu_kernel<float, 3, SLOT_REP>;
    case 5: return (void*)dmumu_kernel<float, 5, SLOT_REP>;
    case 6: return (void*)dmumu_kernel<float, 6, SLOT_REP>;
    case 7: return (void*)dmumu_kernel<float, 7, SLOT_REP>;
    case 4: return dmumu_fn_ns<MuT, 4>(mode);
    default: return dmumu_fn_ns<MuT, 8>(mode);
    }
}

// Device memory of the partials: the context's grow-only scratch, or a fixed array.
struct PartSource {
    pt_ctx* ctx;
    char* fixed;        // null: the context's scratch
    size_t fixed_bytes;
};

size_t part_bytes(int64_t grid, int nl, int n_bins)
{
    return 3 * up16((size_t)grid * nl * n_bins * 8) + up16(sizeof(WelfordPart) * (size_t)grid * nl);
}

template <class Launch>
void set_parts(Launch& L, char* base, int64_t grid, int nl, int n_bins)
{
    const size_t cell = up16((size_t)grid * nl * n_bins * 8);
    L.part_cnt = (unsigned long long*)base;
    L.part_sd = (double*)(base + cell);
    L.part_sd2 = (double*)(base + 2 * cell);
    L.part_w = (WelfordPart*)(base + 3 * cell);
}

int finalize(const DmumuArgs& a, const unsigned long long* cnt, const double* sd, const double* sd2,
             const WelfordPart* w, int grid, int nl, int lag0, cudaStream_t s)
{
    const int cells = (nl * a.n_bins + kWarp - 1) / kWarp;
    dmumu_finalize_kernel<<<cells + nl, kWarp * kFinRows, 0, s>>>(cnt, sd, sd2, w, grid, nl, a.n_bins, lag0, cells,
                                                                  a.counts, a.sum_d, a.sum_d2, a.w_count, a.w_mean,
                                                                  a.w_m2, a.pair_ss, a.pair_n);
    PT_CHECK_LAUNCH("dmumu_finalize_kernel");
    return PT_OK;
}

// D_mumu over a mu chunk, element (p, s) at mu[p * sp + s * ss]
template <typename MuT>
int run_dmumu_t(const PartSource& src, const DmumuArgs& a, const MuT* mu, int64_t sp, int64_t ss, cudaStream_t s,
                int packed = 0)
{
    pt_ctx* ctx = src.ctx;
    if (a.n <= 0 || a.n_lags <= 0) return PT_OK;
    if (a.n_bins < 1 || a.n_bins > 4096) return fail(PT_ERR_ARG, "n_bins must be in [1, 4096]");
    if (a.nsave < 1) return fail(PT_ERR_ARG, "nsave must be positive");
    if (a.nsave >= INT32_MAX) return fail(PT_ERR_ARG, "nsave must be below 2^31");
    const DmumuLimits lim = dmumu_limits(a, sizeof(MuT));
    int max_smem = 0;
    cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, ctx->device);
    if (lim.fixed > (size_t)max_smem)
        return fail(PT_ERR_CUDA, "n_bins is too large for the on-chip (lag, bin) sums");
    if (src.fixed && lim.fixed + lim.slot > kDmumuBudget)
        return fail(PT_ERR_ARG, "pt_dmumu_accumulate_device_noalloc: nsave = " + std::to_string(a.nsave) +
                                    " is too long for on-chip staging with " + std::to_string(a.n_bins) +
                                    " bins; use pt_dmumu_accumulate_device");
    for (int lag0 = 0; lag0 < a.n_lags; lag0 += lim.nl_cap) {
        const int nl = std::min(lim.nl_cap, a.n_lags - lag0);
        DmumuShape h{};
        void* kfn;
        int threads, tile = 0, per_sm = 1;
        size_t smem;
        int64_t blocks;
        if (a.injection) {
            tile = 128;
            while (tile > 32 && dmumu_inj_fixed(nl, a.n_bins, sizeof(MuT), tile).total > (size_t)max_smem / 2) tile /= 2;
            while (tile > 1 && dmumu_inj_fixed(nl, a.n_bins, sizeof(MuT), tile).total > (size_t)max_smem) tile /= 2;
            smem = dmumu_inj_fixed(nl, a.n_bins, sizeof(MuT), tile).total;
            kfn = (void*)dmumu_injection_kernel<MuT>;
            threads = kInjThreads;
            blocks = (a.n + tile - 1) / tile;
        } else {
            h = dmumu_shape(a.n, a.nsave, nl, a.n_bins, sizeof(MuT), (size_t)max_smem, ctx->num_sms);
            kfn = dmumu_fn<MuT>(h.mode, h.ns);
            smem = h.fixed.total + (size_t)h.ppc * h.slot.total;
            threads = h.ppc * h.groups * h.parts * kWarp;
            blocks = (a.n + h.ppc - 1) / h.ppc;
        }
        PT_CUDA(allow_smem(kfn, smem));
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kfn, threads, smem);
        // one CTA per SM where the series are in global memory, as the bound of the
        // scratch that callers are given counts on (registers allow no second one anyway)
        if (!a.injection && h.mode == SLOT_GLOBAL) per_sm = 1;
        blocks = std::min<int64_t>(blocks, (int64_t)ctx->num_sms * std::max(1, per_sm));
        if (src.fixed) {
            const size_t per_cta = (size_t)nl * a.n_bins * 24 + sizeof(WelfordPart) * (size_t)nl + 64;
            const int64_t cap = (int64_t)((src.fixed_bytes - 1024) / per_cta);
            if (cap < 1)
                return fail(PT_ERR_ARG, "pt_dmumu_accumulate_device_noalloc: n_lags x n_bins too large for the " +
                                            std::to_string(src.fixed_bytes >> 20) + " MiB fixed scratch");
            blocks = std::min(blocks, cap);
        }
        const int grid = (int)std::max<int64_t>(1, blocks);
        const size_t gslot = h.mode == SLOT_GLOBAL && !a.injection
                                 ? up16(sizeof(MuT) * (size_t)a.nsave) + up16(sizeof(uint32_t) * (size_t)a.nsave)
                                 : 0;
        const size_t pb = part_bytes(grid, nl, a.n_bins);
        const size_t bytes = pb + (size_t)grid * h.ppc * gslot;
        void* scratch = src.fixed;
        if (!src.fixed) {
            int rc = scratch_get(ctx, 0, bytes, &scratch);
            if (rc) return rc;
        } else if (bytes > src.fixed_bytes) {
            return fail(PT_ERR_ARG, "internal: no-alloc scratch overflow");
        }
        // a CTA counts in 32 bits: particles per launch bounded by 2^32 starts per CTA
        int64_t step = a.n;
        if (!a.injection)
            step = std::max<int64_t>(1, (int64_t)((uint64_t)UINT32_MAX / (uint64_t)a.nsave) / 2) * grid;
        for (int64_t p0 = 0; p0 < a.n; p0 += step) {
            const int64_t m = std::min(step, a.n - p0);
            const unsigned long long* cnt;
            const double *sd, *sd2;
            const WelfordPart* w;
            if (a.injection) {
                DmumuInjection L{};
                L.mu = mu + p0 * sp; L.sp = sp; L.ss = ss;
                L.packed = packed; L.first = 1 + lag0;
                L.n = m; L.nsave = a.nsave; L.lags = a.lags + lag0; L.nl = nl;
                L.edges = a.edges; L.n_bins = a.n_bins; L.bin_abs = a.bin_abs; L.tile = tile;
                set_parts(L, (char*)scratch, grid, nl, a.n_bins);
                dmumu_injection_kernel<MuT><<<grid, threads, smem, s>>>(L);
                PT_CHECK_LAUNCH("dmumu_injection_kernel");
                cnt = L.part_cnt; sd = L.part_sd; sd2 = L.part_sd2; w = L.part_w;
            } else {
                DmumuLaunch L{};
                L.mu = mu + p0 * sp; L.sp = sp; L.ss = ss;
                L.n = m; L.nsave = a.nsave; L.lags = a.lags + lag0; L.nl = nl;
                L.edges = a.edges; L.n_bins = a.n_bins; L.bin_abs = a.bin_abs;
                L.ppc = h.ppc; L.groups = h.groups; L.parts = h.parts;
                L.slot_bytes = (int)h.slot.total;
                L.gslots = gslot ? (char*)scratch + pb : nullptr;
                L.gslot_bytes = gslot;
                set_parts(L, (char*)scratch, grid, nl, a.n_bins);
                void* args[] = {&L};
                PT_CUDA(cudaLaunchKernel(kfn, dim3(grid), dim3(threads), args, smem, s));
                PT_CHECK_LAUNCH("dmumu_kernel");
                cnt = L.part_cnt; sd = L.part_sd; sd2 = L.part_sd2; w = L.part_w;
            }
            int rc = finalize(a, cnt, sd, sd2, w, grid, nl, lag0, s);
            if (rc) return rc;
        }
    }
    return PT_OK;
}

}  // namespace

int run_dmumu(pt_ctx* ctx, const DmumuArgs& a, cudaStream_t s)
{
    return run_dmumu_t<float>(PartSource{ctx, nullptr, 0}, a, a.mu, a.sp, a.ss, s);
}

int run_dmumu_chunk(pt_ctx* ctx, const DmumuArgs& a, const void* mu, int64_t sp, int64_t ss, int f64, int packed,
                    cudaStream_t s)
{
    const PartSource src{ctx, nullptr, 0};
    return f64 ? run_dmumu_t<double>(src, a, (const double*)mu, sp, ss, s, packed)
               : run_dmumu_t<float>(src, a, (const float*)mu, sp, ss, s, packed);
}

}  // namespace pt

// ---------------------------------------------------------------------------
// D_mumu accumulation that allocates nothing.
//
// Some callers cannot let a library allocate device memory: a host that owns
// all device memory through its own pool (the Julia host's CUDA.jl pool, or
// the campaign server's HBM-budget admission) has no way to account for a
// cudaMalloc made behind its back, and cudaFree synchronises the whole
// device, stalling every other stream of a busy GPU.  For them the per-CTA
// partials of the D_mumu kernel live in a fixed, file-scope device array of
// kDmumuNoAllocBytes (16 MiB) that every GPU which loads the library holds
// until the process exits.  The array's device address is looked up once per
// device with cudaGetSymbolAddress (host code cannot use the symbol itself:
// on the host it names a stand-in, not device memory).
// ---------------------------------------------------------------------------
static constexpr size_t kDmumuNoAllocBytes = (size_t)16 << 20;
static __device__ __align__(256) unsigned char g_dmumu_noalloc_scratch[kDmumuNoAllocBytes];

namespace pt {
namespace {

constexpr int kMaxDevices = 64;
std::mutex g_noalloc_mutex;
void* g_noalloc_ptr[kMaxDevices] = {};

// Device address of the fixed scratch on `device` (set up on first use).
int noalloc_scratch(int device, void** out)
{
    if (device < 0 || device >= kMaxDevices) return fail(PT_ERR_ARG, "device index out of range");
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (!g_noalloc_ptr[device]) {
        int prev = 0;
        cudaError_t e = cudaGetDevice(&prev);
        if (e != cudaSuccess) return cuda_fail(e, "cudaGetDevice");
        e = cudaSetDevice(device);
        if (e != cudaSuccess) return cuda_fail(e, "cudaSetDevice");
        void* p = nullptr;
        e = cudaGetSymbolAddress(&p, g_dmumu_noalloc_scratch);
        cudaError_t e2 = cudaSetDevice(prev);
        if (e != cudaSuccess) return cuda_fail(e, "cudaGetSymbolAddress(g_dmumu_noalloc_scratch)");
        if (e2 != cudaSuccess) return cuda_fail(e2, "cudaSetDevice");
        g_noalloc_ptr[device] = p;
    }
    *out = g_noalloc_ptr[device];
    return PT_OK;
}

}  // namespace
}  // namespace pt

extern "C" int pt_dmumu_accumulate_device_noalloc(pt_ctx* ctx, const float* d_mu, int64_t n, int64_t nsave, int64_t sp,
                                                  int64_t ss, const int64_t* d_lags, int n_lags, const double* d_edges,
                                                  int n_bins, int start_mode, int bin_abs, int64_t* d_counts,
                                                  double* d_sum_d, double* d_sum_d2, int64_t* d_w_count,
                                                  double* d_w_mean, double* d_w_m2, double* d_pair_ss,
                                                  int64_t* d_pair_n)
{
    using namespace pt;
    if (!ctx) return fail(PT_ERR_ARG, "ctx is null");
    if (n < 0 || nsave < 1 || n_lags < 0 || n_bins < 1) return fail(PT_ERR_ARG, "bad sizes");
    if (start_mode != PT_START_SLIDING && start_mode != PT_START_INJECTION) return fail(PT_ERR_ARG, "start_mode");
    if (n == 0 || n_lags == 0) return PT_OK;
    if (!(d_mu && d_lags && d_edges && d_counts && d_sum_d && d_sum_d2 && d_w_count && d_w_mean && d_w_m2 &&
          d_pair_ss && d_pair_n))
        return fail(PT_ERR_ARG, "null pointer");
    PT_DEVICE_SCOPE(ctx->device);
    DmumuArgs a{d_mu, n, nsave, sp, ss, d_lags, n_lags, d_edges, n_bins, start_mode == PT_START_INJECTION, bin_abs != 0,
                d_counts, d_sum_d, d_sum_d2, d_w_count, d_w_mean, d_w_m2, d_pair_ss, d_pair_n};
    void* scratch = nullptr;
    const int rc = noalloc_scratch(ctx->device, &scratch);
    if (rc) return rc;
    return run_dmumu_t<float>(PartSource{ctx, (char*)scratch, kDmumuNoAllocBytes}, a, a.mu, a.sp, a.ss, ctx->stream);
}
