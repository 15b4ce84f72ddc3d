// Lag-pair statistics on the device.
//
// D_pp (process_momenta_chunk_dpp_cpu!, src/compute_dpp_full.jl:247-288)
// ---------------------------------------------------------------------
// |p| is computed once per (particle, save) in FP64 and staged on chip; every
// lag's count, sum(dp) and sum(dp^2) are added up there, and the normalised sums
// sum(dp/p0) = sum(dp)/p0 and sum((dp/p0)^2) = sum(dp^2)/p0^2 are formed once per
// lag at the end, which equals the reference's per-pair division up to rounding.
#include <math_constants.h>

#include "exact_mu.cuh"

#include <cstdlib>
#include <cstring>
#include "pt_internal.cuh"

#include <algorithm>
#include <optional>

namespace pt {
namespace {

constexpr int kWarp = 32;

// ------------------------------------------------------------------ D_pp
// momentum_magnitude (src/compute_dpp_full.jl:232-234) with the reference's
// rounding: explicitly rounded products and sums are never contracted into
// FMA, so |p| is bit-identical to the reference's and dp = p_end - p_start
// keeps its last bits.
__device__ __forceinline__ double pmag_exact(float px, float py, float pz)
{
    const double x = (double)px, y = (double)py, z = (double)pz;
    return __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(x, x), __dmul_rn(y, y)), __dmul_rn(z, z)));
}

struct DppPart {
    long long count;
    double sdp, sdp2;
};

constexpr int kDppThreads = 512;
constexpr int kDppWarps = kDppThreads / kWarp;
constexpr int kDppLags = 4;    // lags of a set: |p|[s] is read once for them
constexpr int kDppUnroll = 2;  // starts per lane and pass
constexpr int kDppStage = 4;   // pairs of saves that a thread stages side by side

struct DppLaunch {
    const double* pmag;    // [n][pitch] |p| of this launch's particles
    int64_t n, nsave, pitch;
    const int64_t* lags;
    int nl;
    int ppc;       // particle series per CTA
    int sets;      // lag sets: a divisor or a multiple of the warps
    int qparts;    // warps of a set that share a tile's particles; the others share the starts
    int first;     // 1: set the partials, 0: add to them
    DppPart* part; // [grid][nl]
};

// |p| of particles [p0, p0 + n) at every save, time-fastest: out[p][s], pitch
// doubles per particle.  A block turns kPmagSaves saves of 32 particles: rows of
// 128 bytes in, rows of kPmagSaves doubles out.  A pass of its own because the pair
// kernel holds three series per CTA: reading its particles there took a line per
// save and component for 12 useful bytes, a fifth of that kernel's L1 wavefronts.
// The launches alternate on particle chunks whose |p| stays in L2.
constexpr int kPmagSaves = 32;
__global__ void __launch_bounds__(256) pmag_kernel(const float* __restrict__ mom, int64_t chunk, int64_t nsave,
                                                   int64_t p0, int64_t n, int64_t pitch, double* __restrict__ out)
{
    __shared__ double tile[kWarp][kPmagSaves + 1];
    const int x = threadIdx.x % kWarp, y = threadIdx.x / kWarp;
    const int64_t s0 = (int64_t)blockIdx.x * kPmagSaves;
    for (int64_t b = blockIdx.y; b * kWarp < n; b += gridDim.y) {
        const int64_t q = b * kWarp + x;
        float v[kPmagSaves / 8][3];
#pragma unroll
        for (int i = 0; i < kPmagSaves / 8; ++i) {
            const int64_t s = s0 + y + 8 * i;
            const float* m = mom + 3 * s * chunk + p0 + q;
#pragma unroll
            for (int c = 0; c < 3; ++c) v[i][c] = s < nsave && q < n ? m[c * chunk] : 0.0f;
        }
#pragma unroll
        for (int i = 0; i < kPmagSaves / 8; ++i) tile[x][y + 8 * i] = pmag_exact(v[i][0], v[i][1], v[i][2]);
        __syncthreads();
#pragma unroll
        for (int i = 0; i < kWarp / 8; ++i) {
            const int64_t r = b * kWarp + y + 8 * i;
            if (r < n && s0 + x < nsave) out[r * pitch + s0 + x] = tile[y + 8 * i][x];
        }
        __syncthreads();
    }
}

struct DppFixed {
    size_t sd2, cnt, sorted, idx, nfin, bad, series;
};
__host__ __device__ inline DppFixed dpp_fixed(int sets, int nl, int ppc)
{
    auto a16 = [](size_t v) { return (v + 15) & ~(size_t)15; };
    DppFixed f;
    f.sd2 = (size_t)(sets > kDppWarps ? sets : kDppWarps) * kDppLags * sizeof(double);
    f.cnt = 2 * f.sd2;
    f.sorted = f.cnt + sizeof(unsigned long long) * nl;
    f.idx = f.sorted + sizeof(int) * nl;
    f.nfin = f.idx + sizeof(int) * nl;
    f.bad = f.nfin + sizeof(int) * ppc;
    f.series = a16(f.bad + sizeof(int) * ppc);
    return f;
}

// Starts [s0, s1) against NL lags: p[s + L[k]] - p[s], added to sd[k] and sq[k]; the
// lanes of a pass take the starts from `lane` on, the next pass is `hop` on.
// TEST: only finite differences count (into cnt).  Starts are unsigned: a series may
// hold nearly 2^31 saves, and the loops look a pass past the end.
template <int NL, bool TEST>
__device__ __forceinline__ void dpp_rows(const double* __restrict__ p, unsigned s0, unsigned s1, const int (&L)[kDppLags], int lane, int hop,
                                         double (&sd)[kDppLags], double (&sq)[kDppLags], int (&cnt)[kDppLags])
{
    auto pair = [&](double ps, double pe, int k) {
        double d = pe - ps;
        if constexpr (TEST) {
            const bool ok = isfinite(d);
            d = ok ? d : 0.0;
            cnt[k] += (int)ok;
        }
        sd[k] += d;
        sq[k] = fma(d, d, sq[k]);
    };
    unsigned s = s0 + lane;
    for (; s + (kDppUnroll - 1) * kWarp < s1; s += hop) {
        double ps[kDppUnroll], pe[kDppUnroll][NL];
#pragma unroll
        for (int u = 0; u < kDppUnroll; ++u) {
            ps[u] = p[s + u * kWarp];
#pragma unroll
            for (int k = 0; k < NL; ++k) pe[u][k] = p[s + L[k] + u * kWarp];
        }
#pragma unroll
        for (int u = 0; u < kDppUnroll; ++u)
#pragma unroll
            for (int k = 0; k < NL; ++k) pair(ps[u], pe[u][k], k);
    }
    if (s < s1) {  // at most the last pass of a lane is not whole
        const double ps = p[s];
#pragma unroll
        for (int k = 0; k < NL; ++k) pair(ps, p[s + L[k]], k);
    }
}
static_assert(kDppUnroll == 2, "dpp_rows ends with one start per lane");

// Lags are dealt to sets of at most kDppLags, in the order of their value back and
// forth over the sets, so that the sets have about equal numbers of pairs; a warp
// owns a set (or every 16th), its lanes take consecutive starts, and the lanes' sums
// are added across the warp once per tile of particles.  A warp's 8-byte |p| reads
// are consecutive (no bank conflicts, whatever the lags), and |p|[s] is read once for
// the set's lags.  Up to 32 lags fill fewer sets than there are warps: the sets stay
// full, and 2 to 16 warps share one, by particles or by starts.
//
// A particle whose finite saves are a prefix [0, nfin) needs no test in the pair
// loop: the starts below nfin - L are exactly lag L's pairs, so a set runs its
// lags together up to the longest one's end, the others on to the next one's, and
// so on, and the count of a lag is max(0, nfin - L).  Other particles take the same
// loops up to nsave - L with a finite test per pair.
//
// A warp's sums have one writer, and the warps of a set and the CTAs are added in
// order: the result is deterministic.
//
// Bound by shared-memory bandwidth: 8 bytes per pair and 8 per start and set,
// about 2.6 cycles of the SM's 128 B/clk per 32 pairs, with the FP64 pipe at 1.5.
// Two CTAs per SM, so that one's staging runs under the other's pairs.
// 65,536 x 4001 saves x 55 lags with 16 energy snapshots and histograms: 8.45 ms
// with two lags per pass, a finite test per pair and the reads of the momenta in
// this kernel; 5.60 ms now (0.85 ms of it in pmag_kernel).  With few lags or short
// series the staging counts: a series at a time, with the finite saves counted, it
// is a chain of load latencies.  65,536 x 201 saves, 1 and 18 lags: 0.45 and 0.50 ms
// that way with one lag per warp, 0.18 and 0.28 now (0.06 in pmag_kernel); x 801
// saves, 4 lags: 0.74 and 0.45.
template <bool SMEM_SLOTS>
__global__ void __launch_bounds__(kDppThreads, 2) dpp_kernel(DppLaunch a)
{
    extern __shared__ __align__(16) unsigned char smem[];
    const int nl = a.nl, nsave = (int)a.nsave, ppc = a.ppc, sets = a.sets;
    const DppFixed F = dpp_fixed(sets, nl, ppc);
    double* acc_sd = (double*)smem;  // [part][set][kDppLags]
    double* acc_sd2 = (double*)(smem + F.sd2);
    unsigned long long* acc_cnt = (unsigned long long*)(smem + F.cnt);  // [lag, by value]
    int* s_lag = (int*)(smem + F.sorted);  // ascending; nsave where no pair exists
    int* s_idx = (int*)(smem + F.idx);     // index of the lag in a.lags
    int* s_nfin = (int*)(smem + F.nfin);   // first non-finite save
    int* s_bad = (int*)(smem + F.bad);     // saves that are not finite
    double* series = (double*)(smem + F.series);  // [ppc][pitch]
    for (int i = threadIdx.x; i < max(sets, kDppWarps) * kDppLags; i += blockDim.x) acc_sd[i] = acc_sd2[i] = 0.0;
    for (int i = threadIdx.x; i < nl; i += blockDim.x) {
        acc_cnt[i] = 0ull;
        auto value = [&](int q) {  // the range test in 64 bits, before the narrowing
            const int64_t v = a.lags[q];
            return v < 1 || v >= a.nsave ? nsave : (int)v;  // lag >= nsteps -> skipped
        };
        const int L = value(i);
        int rank = 0;
        for (int q = 0; q < nl; ++q) {
            const int Lq = value(q);
            rank += Lq < L || (Lq == L && q < i);
        }
        s_lag[rank] = L;
        s_idx[rank] = i;
    }
    __syncthreads();  // a CTA without a tile goes straight to the partials
    const int warp = threadIdx.x / kWarp, lane = threadIdx.x % kWarp;
    // lag k of a set, by value: rows of `sets` lags dealt forth and back
    auto dealt = [&](int set, int k) { return k * sets + (k & 1 ? sets - 1 - set : set); };
    // fewer sets than warps: `parts` warps share a set
    const int across = min(sets, kDppWarps), parts = kDppWarps / across, part = warp / across;
    const int from_start = part / a.qparts * (kDppUnroll * kWarp) + lane;
    const int hop = parts / a.qparts * (kDppUnroll * kWarp);
    const int64_t tiles = (a.n + ppc - 1) / ppc;
    for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int64_t p0 = tile * ppc;
        const int np = (int)min(a.n - p0, (int64_t)ppc);
        const double* from = a.pmag + p0 * a.pitch;
        for (int i = threadIdx.x; i < ppc; i += blockDim.x) {
            s_nfin[i] = nsave;
            s_bad[i] = 0;
        }
        __syncthreads();
        // the tile is one run of memory, copied two saves at a time (the pitch is even
        // and the rows 16-byte aligned) whatever the length of a series; which
        // particle a save belongs to matters only where it is not finite
        const int half = (int)(a.pitch / 2), all = np * half;
        const double2* row = (const double2*)from;
        for (int i0 = warp * kWarp + lane; i0 - lane < all; i0 += kDppStage * kDppThreads) {
            double2 v[kDppStage];
#pragma unroll
            for (int k = 0; k < kDppStage; ++k) {
                const int i = i0 + k * kDppThreads;
                v[k] = i < all ? row[i] : make_double2(0.0, 0.0);
            }
#pragma unroll
            for (int k = 0; k < kDppStage; ++k) {
                const int i = i0 + k * kDppThreads;
                if (SMEM_SLOTS && i < all) ((double2*)series)[i] = v[k];
                const bool bx = !isfinite(v[k].x), by = !isfinite(v[k].y);
                if (!__any_sync(0xffffffffu, bx || by)) continue;
                const int q = min(i, all - 1) / half, s = 2 * (i - q * half);
                const bool y = by && s + 1 < nsave;  // the pad of an odd series is no save
                // the lanes of a particle add their counts up first
                const unsigned same = __match_any_sync(0xffffffffu, q);
                const int n = __reduce_add_sync(same, (int)bx + (int)y);
                const int first = __reduce_min_sync(same, bx ? s : (y ? s + 1 : nsave));
                if (n > 0 && lane == __ffs(same) - 1) {
                    atomicAdd(&s_bad[q], n);
                    atomicMin(&s_nfin[q], first);
                }
            }
        }
        __syncthreads();
        for (int l = threadIdx.x; l < nl; l += blockDim.x) {
            long long c = 0;
            for (int q = 0; q < np; ++q)
                if (nsave - s_bad[q] == s_nfin[q]) c += max(0, s_nfin[q] - s_lag[l]);
            if (c > 0) atomicAdd(&acc_cnt[l], (unsigned long long)c);
        }
        for (int set = warp % across; set < sets; set += kDppWarps) {
            int L[kDppLags], cnt[kDppLags];
            double sd[kDppLags], sq[kDppLags];
#pragma unroll
            for (int k = 0; k < kDppLags; ++k) {
                const int l = dealt(set, k);
                L[k] = l < nl ? s_lag[l] : nsave;
                cnt[k] = 0;
                sd[k] = sq[k] = 0.0;
            }
            for (int q = part % a.qparts; q < np; q += a.qparts) {
                const bool prefix = nsave - s_bad[q] == s_nfin[q];
                const int end = prefix ? s_nfin[q] : nsave;
                int lim[kDppLags];  // falls with k
#pragma unroll
                for (int k = 0; k < kDppLags; ++k) lim[k] = max(0, end - L[k]);
                const double* p = (SMEM_SLOTS ? (const double*)series : from) + q * a.pitch;
                if (prefix) {
                    dpp_rows<4, false>(p, 0, lim[3], L, from_start, hop, sd, sq, cnt);
                    dpp_rows<3, false>(p, lim[3], lim[2], L, from_start, hop, sd, sq, cnt);
                    dpp_rows<2, false>(p, lim[2], lim[1], L, from_start, hop, sd, sq, cnt);
                    dpp_rows<1, false>(p, lim[1], lim[0], L, from_start, hop, sd, sq, cnt);
                } else {
                    dpp_rows<4, true>(p, 0, lim[3], L, from_start, hop, sd, sq, cnt);
                    dpp_rows<3, true>(p, lim[3], lim[2], L, from_start, hop, sd, sq, cnt);
                    dpp_rows<2, true>(p, lim[2], lim[1], L, from_start, hop, sd, sq, cnt);
                    dpp_rows<1, true>(p, lim[1], lim[0], L, from_start, hop, sd, sq, cnt);
                }
            }
#pragma unroll
            for (int k = 0; k < kDppLags; ++k) {
#pragma unroll
                for (int o = kWarp / 2; o > 0; o >>= 1) {
                    sd[k] += __shfl_xor_sync(0xffffffffu, sd[k], o);
                    sq[k] += __shfl_xor_sync(0xffffffffu, sq[k], o);
                    cnt[k] += __shfl_xor_sync(0xffffffffu, cnt[k], o);
                }
                if (lane == 0) {
                    acc_sd[(part * sets + set) * kDppLags + k] += sd[k];
                    acc_sd2[(part * sets + set) * kDppLags + k] += sq[k];
                    const int l = dealt(set, k);
                    if (l < nl && cnt[k] > 0) atomicAdd(&acc_cnt[l], (unsigned long long)cnt[k]);
                }
            }
        }
        __syncthreads();
    }
    for (int i = threadIdx.x; i < sets * kDppLags; i += blockDim.x) {
        const int l = dealt(i / kDppLags, i % kDppLags);
        if (l >= nl) continue;
        DppPart& out = a.part[(int64_t)blockIdx.x * nl + s_idx[l]];
        DppPart r{(long long)acc_cnt[l], 0.0, 0.0};
        for (int q = 0; q < parts; ++q) {
            r.sdp += acc_sd[q * sets * kDppLags + i];
            r.sdp2 += acc_sd2[q * sets * kDppLags + i];
        }
        if (!a.first) {
            r.count += out.count;
            r.sdp += out.sdp;
            r.sdp2 += out.sdp2;
        }
        out = r;
    }
}

// One block per lag: threads add the CTAs t, t + 256, ... and a tree adds the
// threads, a fixed order.  (One thread per lag walking all CTAs took 48 us.)
constexpr int kDppFinThreads = 256;
__global__ void __launch_bounds__(kDppFinThreads)
    dpp_finalize_kernel(const DppPart* __restrict__ part, int grid, int nl, int lag0, double p0, int64_t* counts,
                        double* sdp, double* sdp2, double* sdn, double* sdn2)
{
    __shared__ DppPart sh[kDppFinThreads];
    const int t = blockIdx.x;
    DppPart r{0, 0, 0};
    for (int g = threadIdx.x; g < grid; g += kDppFinThreads) {
        const DppPart q = part[(int64_t)g * nl + t];
        r.count += q.count; r.sdp += q.sdp; r.sdp2 += q.sdp2;
    }
    sh[threadIdx.x] = r;
    __syncthreads();
    for (int w = kDppFinThreads / 2; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w) {
            const DppPart q = sh[threadIdx.x + w];
            DppPart& m = sh[threadIdx.x];
            m.count += q.count; m.sdp += q.sdp; m.sdp2 += q.sdp2;
        }
        __syncthreads();
    }
    if (threadIdx.x != 0) return;
    r = sh[0];
    const int l = lag0 + t;
    counts[l] += r.count;
    sdp[l] += r.sdp;
    sdp2[l] += r.sdp2;
    sdn[l] += r.sdp / p0;
    sdn2[l] += r.sdp2 / p0 / p0;
}

// ------------------------------------------------------------------ energies
// kinetic_energy_gev_from_pmag (dpp:236-240)
__device__ __forceinline__ double kinetic_gev(double pmag)
{
    if (!isfinite(pmag)) return NAN;
    const double gev_to_j = 1.0e9 * 1.602176634e-19;
    const double r = __ddiv_rn(pmag, M_P * C_LIGHT);
    const double gamma = __dsqrt_rn(__dadd_rn(1.0, __dmul_rn(r, r)));
    return __ddiv_rn(__dmul_rn(__dmul_rn(__dadd_rn(gamma, -1.0), M_P), C_LIGHT * C_LIGHT), gev_to_j);
}

// snapshot indices outside [0, nsave) (possible for the device entry point,
// whose indices the host cannot see) give NaN instead of a stray read
__global__ void energy_snap_kernel(const float* __restrict__ mom, int64_t chunk, int64_t nsave,
                                   const int64_t* __restrict__ snaps, int n_snap, int64_t offset,
                                   double* __restrict__ out)
{
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= chunk * n_snap) return;
    const int64_t p = t % chunk;
    const int j = (int)(t / chunk);
    const int64_t sj = snaps[j];
    if (sj < 0 || sj >= nsave) {
        out[(offset + p) * n_snap + j] = NAN;
        return;
    }
    const float* m = mom + sj * 3 * chunk + p;
    out[(offset + p) * n_snap + j] = kinetic_gev(pmag_exact(m[0], m[chunk], m[2 * chunk]));
}

__global__ void energy_hist_kernel(const float* __restrict__ mom, int64_t chunk, int64_t nsave,
                                   const int64_t* __restrict__ snaps, int n_snap, double log_emin, double inv_dlog,
                                   int n_hist, unsigned long long* __restrict__ counts)
{
    extern __shared__ unsigned long long h[];
    for (int i = threadIdx.x; i < n_snap * n_hist; i += blockDim.x) h[i] = 0ull;
    __syncthreads();
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < chunk * n_snap;
         t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t p = t % chunk;
        const int j = (int)(t / chunk);
        const int64_t sj = snaps[j];
        if (sj < 0 || sj >= nsave) continue;  // not a save of this chunk: counted nowhere
        const float* m = mom + sj * 3 * chunk + p;
        const double e = kinetic_gev(pmag_exact(m[0], m[chunk], m[2 * chunk]));
        if (!(e > 0.0) || !isfinite(e)) continue;
        const double f = (log(e) - log_emin) * inv_dlog;
        if (!(f >= 0.0) || f >= (double)n_hist) continue;
        atomicAdd(&h[j * n_hist + (int)f], 1ull);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < n_snap * n_hist; i += blockDim.x)
        if (h[i]) atomicAdd(&counts[i], h[i]);
}

size_t align16(size_t b) { return (b + 15) & ~(size_t)15; }

// (Bx, By, Bz) column-major arrays -> one record per node
template <typename R>
__global__ void interleave_b_kernel(const R* __restrict__ bx, const R* __restrict__ by, const R* __restrict__ bz,
                                    int64_t nodes, exact::Vec4<R>* __restrict__ out)
{
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nodes; i += (int64_t)gridDim.x * blockDim.x)
        out[i] = exact::Vec4<R>{bx[i], by[i], bz[i], R(0)};
}

// (Bx, By, Bz) column-major arrays -> one 8-corner record per cell, indexed
// by the cell's base node (nodes on the last x, y or z plane are no base and
// their records are left unwritten: a sample never reads them).  Thread per
// record: the corner reads of neighbouring threads coalesce, and so do the
// record writes.
template <typename R>
__global__ void cell_b_kernel(const R* __restrict__ bx, const R* __restrict__ by, const R* __restrict__ bz, int64_t nx,
                              int64_t ny, int64_t nz, exact::CellB<R>* __restrict__ out)
{
    const int64_t nodes = nx * ny * nz, sy = nx, sz = nx * ny;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nodes; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t ix = i % nx, iy = (i / nx) % ny, iz = i / sz;
        if (ix >= nx - 1 || iy >= ny - 1 || iz >= nz - 1) continue;
        const int64_t off[8] = {0, 1, sy, 1 + sy, sz, 1 + sz, sy + sz, 1 + sy + sz};
        exact::CellB<R> r;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            r.v[3 * q] = bx[i + off[q]];
            r.v[3 * q + 1] = by[i + off[q]];
            r.v[3 * q + 2] = bz[i + off[q]];
        }
        out[i] = r;
    }
}

// Where phase_space_mu_kernel reads B from.
enum { B_CELLS = 0, B_NODES = 1, B_ARRAYS = 2 };
struct BSource {
    const void* records;   // cell or node records
    const void* arrays[3]; // Bx, By, Bz as they are
};

// mu of particles [p0, p0 + m) at saves save[r] of `rows` (all saves, or save 0
// and the lags'), written time-fastest, mu[p - p0][r].  A block takes 32 particles
// at kPsRows saves: a warp per save, a lane per particle, so that the phase-space
// reads coalesce; the tile is turned in shared memory, so that the writes do, and
// the binning reads whole series.
//
// With cell records a sample's B is one contiguous record (96 bytes in FP32) at a
// random place.  The lanes fetch each other's records: 8 (FP64: 16) lanes copy one
// record to shared memory with 16-byte asynchronous copies, 4 (2) records per warp
// instruction.  The kernel is bound by the L1's queue of requests that miss, one per
// line and instruction: with each lane reading its own record in 32-byte loads that
// queue was full (a third of all stalls) at 41 % of the DRAM bandwidth; now DRAM is
// 75 % busy.  256^3, 65,536 particles x 801 saves, FP32: 3.20 ms, 2.00 ms now.
template <typename R>
constexpr int kPsRows = sizeof(R) == 4 ? 8 : 4;  // 32-byte runs of a particle's mu

__device__ __forceinline__ void copy16_async(void* smem, const void* from)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(from)
                 : "memory");
}

template <typename R, int SRC>
__global__ void __launch_bounds__(kWarp* kPsRows<R>)
    phase_space_mu_kernel(const R* __restrict__ pos, const R* __restrict__ mom, int64_t row, int64_t comp, int64_t p0,
                          int64_t m, int64_t rows, int64_t nsave, const int64_t* __restrict__ lags, BSource B,
                          pt_grid g, int64_t pitch, R* __restrict__ mu)
{
    constexpr int kChunks = 24 * sizeof(R) / 16;                // 16-byte pieces of a record
    constexpr int kLanes = kChunks <= 8 ? 8 : 16;               // lanes that copy one
    constexpr int kRecord = 24 * sizeof(R) + 16;                // padded: a quarter warp's reads hit all banks
    __shared__ __align__(16) unsigned char s_rec[SRC == B_CELLS ? kPsRows<R> * kWarp * kRecord : 16];
    __shared__ R tile[kWarp][kPsRows<R> + 1];
    const int lane = threadIdx.x % kWarp, w = threadIdx.x / kWarp;
    const int64_t blocks_p = (m + kWarp - 1) / kWarp, blocks_r = (rows + kPsRows<R> - 1) / kPsRows<R>;
    for (int64_t t = blockIdx.x; t < blocks_p * blocks_r; t += gridDim.x) {
        const int64_t q = t % blocks_p * kWarp + lane, r0 = t / blocks_p * kPsRows<R>, r = r0 + w;
        int64_t s = r;
        if (lags && r > 0 && r < rows) s = lags[r - 1];  // the injection estimator's rows: save 0, then the lags'
        const bool have = r < rows && q < m && s >= 0 && s < nsave;
        R v = R(NAN), x[3], p[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            x[k] = have ? pos[s * row + k * comp + p0 + q] : R(NAN);
            p[k] = have ? mom[s * row + k * comp + p0 + q] : R(NAN);
        }
        const bool in = exact::phase_space_inside<R>(x[0], x[1], x[2], p[0], p[1], p[2], g);
        if constexpr (SRC == B_CELLS) {
            exact::Cell<R> c{};
            c.base = -1;
            if (in)
                c = exact::locate<R>(x[0], x[1], x[2], (R)g.xmin, (R)g.ymin, (R)g.zmin, (R)g.dx, (R)g.dy, (R)g.dz, g.nx,
                                     g.ny, g.nz);
            unsigned char* mine = s_rec + (size_t)w * kWarp * kRecord;
            const int part = lane % kLanes;
#pragma unroll
            for (int k = 0; k < kLanes; ++k) {
                const int owner = k * (kWarp / kLanes) + lane / kLanes;
                const int64_t base = __shfl_sync(0xffffffffu, (long long)c.base, owner);
                if (base >= 0 && part < kChunks)
                    copy16_async(mine + owner * kRecord + 16 * part,
                                 (const char*)B.records + base * (int64_t)sizeof(exact::CellB<R>) + 16 * part);
            }
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncwarp();
            if (in) v = exact::cell_mu<R>((const R*)(mine + lane * kRecord), c, p[0], p[1], p[2]);
        } else if (in) {
            if constexpr (SRC == B_NODES) {
                v = exact::phase_space_mu4<R>(x[0], x[1], x[2], p[0], p[1], p[2], (const exact::Vec4<R>*)B.records, g);
            } else {
                const R* const b[3] = {(const R*)B.arrays[0], (const R*)B.arrays[1], (const R*)B.arrays[2]};
                v = exact::phase_space_mu<R>(x[0], x[1], x[2], p[0], p[1], p[2], b, g);
            }
        }
        tile[lane][w] = v;
        __syncthreads();
        // thread -> (particle, save), saves fastest
        const int tp = threadIdx.x / kPsRows<R>, tr = threadIdx.x % kPsRows<R>;
        const int64_t op = t % blocks_p * kWarp + tp;
        if (op < m && r0 + tr < rows) mu[op * pitch + r0 + tr] = tile[tp][tr];
        __syncthreads();
    }
}

template <typename R>
int run_dmumu_phase_space_t(pt_ctx* ctx, const DmumuArgs& a, const R* pos, const R* mom, int64_t row, int64_t comp,
                            const void* const bfield[3], const pt_grid& g, cudaStream_t s)
{
    using V4 = exact::Vec4<R>;
    using CB = exact::CellB<R>;
    const int64_t nodes = g.nx * g.ny * g.nz;
    // the injection estimator needs save 0 and the lags' saves only
    const int64_t rows = a.injection ? 1 + (int64_t)a.n_lags : a.nsave;
    // mu chunks of at most 1 GiB
    const int64_t per = std::max<int64_t>(1, ((int64_t)1 << 30) / ((int64_t)sizeof(R) * rows));
    const int64_t m_max = std::min<int64_t>(a.n, per);
    const size_t mu_bytes = sizeof(R) * (size_t)m_max * (size_t)rows;
    // B as cell records when they take at most half of the free device
    // memory: a sample then reads one 96-byte (FP32) record instead of 8
    // node records from 4 grid rows, ~4x fewer DRAM bytes on the random
    // gathers of particles in id order; otherwise as node records.  Building
    // the records reads and writes 108 (28) bytes per node, which pays from
    // about half (an eighth) as many samples as nodes; below, the arrays are read
    // as they are.
    const int64_t samples = a.n * rows;
    const size_t cell_bytes = align16(sizeof(CB) * (size_t)nodes);
    int src = samples >= nodes / 2 ? B_CELLS : (samples >= nodes / 8 ? B_NODES : B_ARRAYS);
    // PTB200_PHASE_SPACE_B = "nodes" or "cells" overrides the choice (same results)
    const char* want = std::getenv("PTB200_PHASE_SPACE_B");
    if (want && !std::strcmp(want, "nodes")) {
        src = B_NODES;
    } else if (want && !std::strcmp(want, "cells")) {
        src = B_CELLS;
    } else if (src == B_CELLS && ctx->scratch[4].bytes < cell_bytes + mu_bytes) {
        // (asked only when the context does not hold the memory already: the query
        // can take as long as the whole call)
        size_t free_b = 0, total_b = 0;
        if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess) {
            cudaGetLastError();
            free_b = 0;
        }
        if (cell_bytes + mu_bytes > free_b / 2) src = B_NODES;
    }
    const size_t b_bytes = src == B_CELLS ? cell_bytes : (src == B_NODES ? align16(sizeof(V4) * (size_t)nodes) : 0);
    void* scratch = nullptr;
    int rc = scratch_get(ctx, 4, b_bytes + mu_bytes, &scratch);
    if (rc) return rc;
    R* mu = (R*)((char*)scratch + b_bytes);
    const int gb = (int)std::min<int64_t>((nodes + 255) / 256, (int64_t)ctx->num_sms * 16);
    const R* b[3] = {(const R*)bfield[0], (const R*)bfield[1], (const R*)bfield[2]};
    if (src == B_CELLS) {
        cell_b_kernel<R><<<gb, 256, 0, s>>>(b[0], b[1], b[2], g.nx, g.ny, g.nz, (CB*)scratch);
        PT_CHECK_LAUNCH("cell_b_kernel");
    } else if (src == B_NODES) {
        interleave_b_kernel<R><<<gb, 256, 0, s>>>(b[0], b[1], b[2], nodes, (V4*)scratch);
        PT_CHECK_LAUNCH("interleave_b_kernel");
    }
    const BSource B{scratch, {bfield[0], bfield[1], bfield[2]}};
    const int64_t* lags = a.injection ? a.lags : nullptr;
    for (int64_t p0 = 0; p0 < a.n; p0 += m_max) {
        const int64_t m = std::min(m_max, a.n - p0);
        const int64_t tiles = ((m + kWarp - 1) / kWarp) * ((rows + kPsRows<R> - 1) / kPsRows<R>);
        const int blocks = (int)std::min<int64_t>(tiles, (int64_t)ctx->num_sms * 64);
        const int threads = kWarp * kPsRows<R>;
        if (src == B_CELLS)
            phase_space_mu_kernel<R, B_CELLS><<<blocks, threads, 0, s>>>(pos, mom, row, comp, p0, m, rows, a.nsave, lags,
                                                                         B, g, rows, mu);
        else if (src == B_NODES)
            phase_space_mu_kernel<R, B_NODES><<<blocks, threads, 0, s>>>(pos, mom, row, comp, p0, m, rows, a.nsave, lags,
                                                                         B, g, rows, mu);
        else
            phase_space_mu_kernel<R, B_ARRAYS><<<blocks, threads, 0, s>>>(pos, mom, row, comp, p0, m, rows, a.nsave,
                                                                          lags, B, g, rows, mu);
        PT_CHECK_LAUNCH("phase_space_mu_kernel");
        DmumuArgs c = a;
        c.n = m;
        rc = run_dmumu_chunk(ctx, c, mu, rows, 1, sizeof(R) == 8, a.injection, s);
        if (rc) return rc;
    }
    return PT_OK;
}

}  // namespace

int run_dmumu_phase_space(pt_ctx* ctx, const DmumuArgs& a, const void* pos, const void* mom, int64_t row,
                          int64_t comp, const void* const bfield[3], const pt_grid& g, int f64, cudaStream_t s)
{
    if (a.n <= 0 || a.n_lags <= 0) return PT_OK;
    if (f64) return run_dmumu_phase_space_t<double>(ctx, a, (const double*)pos, (const double*)mom, row, comp, bfield,
                                                    g, s);
    return run_dmumu_phase_space_t<float>(ctx, a, (const float*)pos, (const float*)mom, row, comp, bfield, g, s);
}

int run_dpp(pt_ctx* ctx, const DppArgs& a, cudaStream_t s)
{
    if (a.chunk <= 0 || a.n_lags <= 0) return PT_OK;
    if (a.nsave >= INT32_MAX) return fail(PT_ERR_ARG, "nsave must be below 2^31");
    int max_smem = 0, sm_smem = 0;
    cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, ctx->device);
    cudaDeviceGetAttribute(&sm_smem, cudaDevAttrMaxSharedMemoryPerMultiprocessor, ctx->device);
    const int64_t pitch = (a.nsave + 1) & ~(int64_t)1;
    const size_t series = sizeof(double) * (size_t)pitch;
    const int nl_cap = 32 * 8;
    for (int lag0 = 0; lag0 < a.n_lags; lag0 += nl_cap) {
        const int nl = std::min(nl_cap, a.n_lags - lag0);
        DppLaunch L;
        L.sets = 1;
        while (L.sets < kDppWarps && L.sets * kDppLags < nl) L.sets *= 2;
        if (L.sets == kDppWarps) L.sets *= (nl + kDppWarps * kDppLags - 1) / (kDppWarps * kDppLags);
        // Series on chip when they fit, two CTAs per SM when half of it holds one
        // (the reserved KB per CTA left out).  As many as fit, up to 16, but no
        // more than gives every CTA of the chip a tile.
        const size_t half = std::min<size_t>(max_smem, sm_smem / 2 - 1024);
        auto need = [&](int ppc) { return dpp_fixed(L.sets, nl, ppc).series + (size_t)ppc * series; };
        const bool two = need(1) <= half;
        const bool smem_slots = two || need(1) <= (size_t)max_smem;
        int ppc = 1;
        while (smem_slots && ppc < 16 && (int64_t)ppc * ctx->num_sms * (two ? 2 : 1) < a.chunk &&
               need(ppc + 1) <= (two ? half : (size_t)max_smem))
            ++ppc;
        // the warps of a set share particles or starts, whichever leaves the busiest the
        // fewest passes
        const int parts = std::max(1, kDppWarps / L.sets);
        int64_t least = 0;
        L.qparts = 1;
        for (int q = 1; q <= parts; q *= 2) {
            const int64_t hop = (int64_t)kDppUnroll * kWarp * (parts / q);
            const int64_t passes = ((ppc + q - 1) / q) * ((a.nsave + hop - 1) / hop);
            if (q == 1 || passes <= least) {
                least = passes;
                L.qparts = q;
            }
        }
        const size_t smem = smem_slots ? need(ppc) : dpp_fixed(L.sets, nl, ppc).series;
        void* kfn = smem_slots ? (void*)dpp_kernel<true> : (void*)dpp_kernel<false>;
        PT_CUDA(allow_smem(kfn, smem));
        int per_sm = 1;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kfn, kDppThreads, smem);
        const int64_t ctas = (int64_t)ctx->num_sms * std::max(1, per_sm);
        const int grid = (int)std::max<int64_t>(1, std::min<int64_t>((a.chunk + ppc - 1) / ppc, ctas));
        // |p| chunks: whole rounds of the CTAs, as many as 128 MB hold.  The context's
        // scratch holds the partials and at least one series, 16 MB in all for series
        // below that, so that it does not grow from call to call (its regrowth stalls
        // the device).  What does not fit there is memory of this call, or, where that
        // is not to be had (a nearly full device, a stream capture), more launches on
        // what the scratch holds.
        const int64_t round = (int64_t)grid * ppc;
        const int64_t rounds = std::max<int64_t>(1, (int64_t)(((size_t)128 << 20) / series) / round);
        int64_t step = std::min<int64_t>(a.chunk, round * rounds);
        const size_t part_bytes = (sizeof(DppPart) * (size_t)grid * nl + 255) & ~(size_t)255;
        void* scratch = nullptr;
        int rc = scratch_get(ctx, 1, part_bytes + series, &scratch);
        if (rc) return rc;
        double* pmag = (double*)((char*)scratch + part_bytes);
        const int64_t held = (int64_t)((ctx->scratch[1].bytes - part_bytes) / series);
        std::optional<CallMem> mem;
        if (held < step) {
            mem.emplace(ctx, (size_t)step * series, s);
            if (mem->get()) pmag = (double*)mem->get();
            else step = held >= round ? held / round * round : held;
        }
        L.pmag = pmag; L.nsave = a.nsave; L.pitch = pitch; L.lags = a.lags + lag0; L.nl = nl;
        L.ppc = ppc;
        L.part = (DppPart*)scratch;
        for (int64_t p0 = 0; p0 < a.chunk; p0 += step) {
            L.n = std::min(step, a.chunk - p0);
            L.first = p0 == 0;
            const dim3 pg((unsigned)((a.nsave + kPmagSaves - 1) / kPmagSaves),
                          (unsigned)std::min<int64_t>((L.n + kWarp - 1) / kWarp, 65535));
            pmag_kernel<<<pg, 256, 0, s>>>(a.mom, a.chunk, a.nsave, p0, L.n, pitch, pmag);
            PT_CHECK_LAUNCH("pmag_kernel");
            if (smem_slots) dpp_kernel<true><<<grid, kDppThreads, smem, s>>>(L);
            else dpp_kernel<false><<<grid, kDppThreads, smem, s>>>(L);
            PT_CHECK_LAUNCH("dpp_kernel");
        }
        dpp_finalize_kernel<<<nl, kDppFinThreads, 0, s>>>(L.part, grid, nl, lag0, a.p0, a.counts, a.sdp, a.sdp2,
                                                          a.sdn, a.sdn2);
        PT_CHECK_LAUNCH("dpp_finalize_kernel");
    }
    return PT_OK;
}

int launch_energy_snapshots(const float* mom, int64_t chunk, int64_t nsave, const int64_t* snaps, int n_snap,
                            int64_t offset, double* out, cudaStream_t s)
{
    const int64_t total = chunk * n_snap;
    if (total <= 0) return PT_OK;
    energy_snap_kernel<<<(unsigned)((total + 255) / 256), 256, 0, s>>>(mom, chunk, nsave, snaps, n_snap, offset, out);
    PT_CHECK_LAUNCH("energy_snap_kernel");
    return PT_OK;
}

int launch_energy_histogram(const float* mom, int64_t chunk, int64_t nsave, const int64_t* snaps, int n_snap,
                            double e_min, double e_max, int n_hist, int64_t* counts, cudaStream_t s)
{
    const int64_t total = chunk * n_snap;
    if (total <= 0) return PT_OK;
    const size_t smem = sizeof(unsigned long long) * (size_t)n_snap * n_hist;
    if (smem > 160 * 1024) return fail(PT_ERR_ARG, "n_snap * n_hist too large for the on-chip histogram");
    if (smem > 48 * 1024) PT_CUDA(allow_smem((const void*)energy_hist_kernel, smem));
    const double log_emin = log(e_min);
    const double inv_dlog = (double)n_hist / (log(e_max) - log_emin);
    const int blocks = (int)std::min<int64_t>((total + 255) / 256, 148 * 4);
    energy_hist_kernel<<<blocks, 256, smem, s>>>(mom, chunk, nsave, snaps, n_snap, log_emin, inv_dlog, n_hist,
                                                 (unsigned long long*)counts);
    PT_CHECK_LAUNCH("energy_hist_kernel");
    return PT_OK;
}

}  // namespace pt
