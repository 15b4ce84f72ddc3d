// Lag-pair statistics on the device.
//
// D_pp (process_momenta_chunk_dpp_cpu!, src/compute_dpp_full.jl:247-288)
// ---------------------------------------------------------------------
// Same layout without bins: |p| is computed once per (particle, save) in FP64
// and every lane keeps its lag's count, sum(dp) and sum(dp^2) in registers for
// the whole launch; the normalised sums sum(dp/p0) = sum(dp)/p0 and
// sum((dp/p0)^2) = sum(dp^2)/p0^2 are formed once per lag at the end, which
// equals the reference's per-pair division up to rounding.
#include <math_constants.h>

#include "exact_mu.cuh"

#include <cstdlib>
#include <cstring>
#include "pt_internal.cuh"

#include <algorithm>

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

struct DppLaunch {
    const float* mom;
    int64_t chunk, nsave;
    const int64_t* lags;
    int nl;
    double p0;
    int ppc, wps;  // particle slots per CTA, warps per slot
    size_t slot_bytes;
    char* gslots;
    DppPart* part;  // [grid][nl]
};

// Warps = (particle slot, lag subset): warp w of a slot owns lags w, w + wps,
// w + 2 wps, ... and takes kDppLags of them at a time; its lanes take the
// starts s = lane, lane + 32, ...  A warp's 8-byte |p| reads are then
// consecutive (no shared-memory bank conflicts, whatever the lags), and
// |p|[s] is read once for the lags of a pass.  The series of a slot holds |p| at saves 0..nsave-1 and
// NaN at index nsave, so the end of a pair past the series reads NaN (an
// invalid pair) with no bounds test.  A lag's sums are warp-reduced once per
// particle and added by lane 0 into the slot's accumulator for that lag (one
// writer per (slot, lag)); the CTA adds its slots in slot order at the end.
// lags of a warp per pass over the starts (|p|[s] read once for them); 4 was
// measured slower: a pass runs to the range of its smallest lag
constexpr int kDppLags = 2;

template <bool SMEM_SLOTS>
__global__ void __launch_bounds__(1024) dpp_kernel(DppLaunch a)
{
    extern __shared__ __align__(16) unsigned char smem[];
    // shared layout: acc[ppc][nl] | slots (when on chip)
    DppPart* acc = (DppPart*)smem;
    const size_t acc_bytes = ((size_t)a.ppc * a.nl * sizeof(DppPart) + 15) & ~(size_t)15;
    unsigned char* slot_base =
        SMEM_SLOTS ? smem + acc_bytes : (unsigned char*)(a.gslots + (size_t)blockIdx.x * a.ppc * a.slot_bytes);
    for (int i = threadIdx.x; i < a.ppc * a.nl; i += blockDim.x) acc[i] = DppPart{0, 0.0, 0.0};
    const int warp = threadIdx.x / kWarp, lane = threadIdx.x % kWarp;
    const int slot = warp / a.wps, w = warp % a.wps;
    const int nsave = (int)a.nsave;  // nsave < 2^31
    double* series = (double*)(slot_base + (size_t)slot * a.slot_bytes);
    const int64_t tiles = (a.chunk + a.ppc - 1) / a.ppc;
    __syncthreads();
    for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        // cooperative staging: thread t -> (save, particle slot)
        const int64_t p0i = tile * a.ppc;
        const int np = (int)(a.chunk - p0i < (int64_t)a.ppc ? a.chunk - p0i : (int64_t)a.ppc);
        for (int64_t t = threadIdx.x; t < (int64_t)np * (a.nsave + 1); t += blockDim.x) {
            const int sl = (int)(t % np);
            const int64_t s = t / np;
            double v = CUDART_NAN;  // the pad at index nsave
            if (s < a.nsave) {
                const float* m = a.mom + s * 3 * a.chunk + p0i + sl;
                v = pmag_exact(m[0], m[a.chunk], m[2 * a.chunk]);
            }
            ((double*)(slot_base + (size_t)sl * a.slot_bytes))[s] = v;
        }
        __syncthreads();
        if (slot < np) {
            // |p| >= 0 or NaN or +inf, so pe - ps is finite exactly when both
            // ends are finite; an invalid pair adds 0 (branch-free), which
            // leaves the sums unchanged.  The normalised sums are sum(d)/p0
            // and sum(d^2)/p0^2, formed once per lag in dpp_finalize_kernel.
            for (int l0 = w; l0 < a.nl; l0 += kDppLags * a.wps) {
                int L[kDppLags], cnt[kDppLags];
                double sd[kDppLags], sq[kDppLags];
                int lmin = nsave;
#pragma unroll
                for (int k = 0; k < kDppLags; ++k) {
                    const int l = l0 + k * a.wps;
                    // the range test in 64 bits, before the narrowing
                    const int64_t v64 = l < a.nl ? a.lags[l] : a.nsave;
                    const int v = (v64 < 1 || v64 >= a.nsave) ? nsave : (int)v64;  // lag >= nsteps -> skipped
                    L[k] = v;
                    lmin = min(lmin, v);
                    cnt[k] = 0;
                    sd[k] = 0.0;
                    sq[k] = 0.0;
                }
                const int lim = nsave - lmin;
                for (int s = lane; s < lim; s += kWarp) {
                    const double ps = series[s];
#pragma unroll
                    for (int k = 0; k < kDppLags; ++k) {
                        const double pe = series[min((unsigned)s + (unsigned)L[k], (unsigned)nsave)];
                        double d = pe - ps;
                        const bool ok = isfinite(d);
                        d = ok ? d : 0.0;
                        cnt[k] += (int)ok;
                        sd[k] += d;
                        sq[k] = fma(d, d, sq[k]);
                    }
                }
#pragma unroll
                for (int k = 0; k < kDppLags; ++k) {
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) {
                        cnt[k] += __shfl_xor_sync(0xffffffffu, cnt[k], o);
                        sd[k] += __shfl_xor_sync(0xffffffffu, sd[k], o);
                        sq[k] += __shfl_xor_sync(0xffffffffu, sq[k], o);
                    }
                    const int l = l0 + k * a.wps;
                    if (lane == 0 && l < a.nl) {
                        DppPart& A = acc[slot * a.nl + l];
                        A.count += cnt[k]; A.sdp += sd[k]; A.sdp2 += sq[k];
                    }
                }
            }
        }
        __syncthreads();
    }
    // CTA epilogue: slots added in slot order
    for (int l = threadIdx.x; l < a.nl; l += blockDim.x) {
        DppPart r{0, 0, 0};
        for (int sl = 0; sl < a.ppc; ++sl) {
            const DppPart v = acc[sl * a.nl + l];
            r.count += v.count; r.sdp += v.sdp; r.sdp2 += v.sdp2;
        }
        a.part[(int64_t)blockIdx.x * a.nl + l] = r;
    }
}

__global__ void dpp_finalize_kernel(const DppPart* __restrict__ part, int grid, int nl, int lag0, double p0,
                                    int64_t* counts, double* sdp, double* sdp2, double* sdn, double* sdn2)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nl) return;
    DppPart r{0, 0, 0};
    for (int g = 0; g < grid; ++g) {
        const DppPart q = part[(int64_t)g * nl + t];
        r.count += q.count; r.sdp += q.sdp; r.sdp2 += q.sdp2;
    }
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

// mu of particles [p0, p0 + m) at every save, written [s][p - p0] (particle
// fastest, like the device mu cache); one thread per (particle, save),
// particles fastest so that the phase-space reads coalesce.  B comes from
// cell records (CELLS) or node records.
template <typename R, bool CELLS>
__global__ void __launch_bounds__(256) phase_space_mu_kernel(const R* __restrict__ pos, const R* __restrict__ mom,
                                                             int64_t row, int64_t comp, int64_t p0, int64_t m,
                                                             int64_t nsave, const void* __restrict__ Bsrc, pt_grid g,
                                                             R* __restrict__ mu)
{
    const int64_t total = m * nsave;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t q = t % m, s = t / m;
        const R* P = pos + s * row + p0 + q;
        const R* M = mom + s * row + p0 + q;
        if constexpr (CELLS)
            mu[s * m + q] = exact::phase_space_mu_cell<R>(P[0], P[comp], P[2 * comp], M[0], M[comp], M[2 * comp],
                                                          (const exact::CellB<R>*)Bsrc, g);
        else
            mu[s * m + q] = exact::phase_space_mu4<R>(P[0], P[comp], P[2 * comp], M[0], M[comp], M[2 * comp],
                                                      (const exact::Vec4<R>*)Bsrc, g);
    }
}

template <typename R>
int run_dmumu_phase_space_t(pt_ctx* ctx, const DmumuArgs& a, const R* pos, const R* mom, int64_t row, int64_t comp,
                            const void* const bfield[3], const pt_grid& g, cudaStream_t s)
{
    using V4 = exact::Vec4<R>;
    using CB = exact::CellB<R>;
    const int64_t nodes = g.nx * g.ny * g.nz;
    // mu chunks of at most 1 GiB
    const int64_t per = std::max<int64_t>(1, ((int64_t)1 << 30) / ((int64_t)sizeof(R) * a.nsave));
    const int64_t m_max = std::min<int64_t>(a.n, per);
    const size_t mu_bytes = sizeof(R) * (size_t)m_max * (size_t)a.nsave;
    // B as cell records when they take at most half of the free device
    // memory: a sample then reads one 96-byte (FP32) record instead of 8
    // node records from 4 grid rows, ~4x fewer DRAM bytes on the random
    // gathers of particles in id order; otherwise as node records
    size_t free_b = 0, total_b = 0;
    if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess) {
        cudaGetLastError();
        free_b = 0;
    }
    const size_t cell_bytes = align16(sizeof(CB) * (size_t)nodes);
    bool cells = cell_bytes + mu_bytes <= free_b / 2;
    // PTB200_PHASE_SPACE_B = "nodes" or "cells" overrides the choice (same results)
    if (const char* e = std::getenv("PTB200_PHASE_SPACE_B")) {
        if (!std::strcmp(e, "nodes")) cells = false;
        else if (!std::strcmp(e, "cells")) cells = true;
    }
    const size_t b_bytes = cells ? cell_bytes : align16(sizeof(V4) * (size_t)nodes);
    void* scratch = nullptr;
    int rc = scratch_get(ctx, 4, b_bytes + mu_bytes, &scratch);
    if (rc) return rc;
    R* mu = (R*)((char*)scratch + b_bytes);
    const int gb = (int)std::min<int64_t>((nodes + 255) / 256, (int64_t)ctx->num_sms * 16);
    if (cells) {
        cell_b_kernel<R><<<gb, 256, 0, s>>>((const R*)bfield[0], (const R*)bfield[1], (const R*)bfield[2], g.nx, g.ny,
                                            g.nz, (CB*)scratch);
        PT_CHECK_LAUNCH("cell_b_kernel");
    } else {
        interleave_b_kernel<R><<<gb, 256, 0, s>>>((const R*)bfield[0], (const R*)bfield[1], (const R*)bfield[2], nodes,
                                                  (V4*)scratch);
        PT_CHECK_LAUNCH("interleave_b_kernel");
    }
    for (int64_t p0 = 0; p0 < a.n; p0 += m_max) {
        const int64_t m = std::min(m_max, a.n - p0);
        const int64_t total = m * a.nsave;
        const int blocks = (int)std::min<int64_t>((total + 255) / 256, (int64_t)ctx->num_sms * 32);
        if (cells)
            phase_space_mu_kernel<R, true><<<blocks, 256, 0, s>>>(pos, mom, row, comp, p0, m, a.nsave, scratch, g, mu);
        else
            phase_space_mu_kernel<R, false><<<blocks, 256, 0, s>>>(pos, mom, row, comp, p0, m, a.nsave, scratch, g, mu);
        PT_CHECK_LAUNCH("phase_space_mu_kernel");
        DmumuArgs c = a;
        c.n = m;
        rc = run_dmumu_chunk(ctx, c, mu, 1, m, sizeof(R) == 8, s);
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
    int max_smem = 0;
    cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, ctx->device);
    const size_t budget = (size_t)std::min(max_smem, 200 * 1024);
    if (a.nsave >= INT32_MAX) return fail(PT_ERR_ARG, "nsave must be below 2^31");
    const size_t slot_bytes = align16(sizeof(double) * (size_t)(a.nsave + 1));  // + NaN pad
    const int nl_cap = 32 * 8;
    for (int lag0 = 0; lag0 < a.n_lags; lag0 += nl_cap) {
        const int nl = std::min(nl_cap, a.n_lags - lag0);
        // particle slots per CTA (series on chip when they fit) and warps per
        // slot (each takes ceil(nl / wps) lags, two at a time)
        const size_t acc_per_slot = sizeof(DppPart) * (size_t)nl;
        bool smem_slots = align16(acc_per_slot) + slot_bytes <= budget;
        // the most warps per CTA (at most 32), the larger ppc among equals:
        // at 55 lags and room for five series, 4 slots x 8 warps measured
        // 1.45e12 lag-pairs/s against 1.32e12 for 5 x 6
        const int max_ppc = smem_slots ? (int)std::min<size_t>(budget / (slot_bytes + acc_per_slot), 8) : 4;
        const int lag_sets = (nl + kDppLags - 1) / kDppLags;
        int ppc = 1, wps = 1, best = 0;
        for (int c = 1; c <= std::max(1, max_ppc); ++c) {
            const int w = std::max(1, std::min(32 / c, lag_sets));
            if (c * w >= best) {
                best = c * w;
                ppc = c;
                wps = w;
            }
        }
        const int threads = ppc * wps * kWarp;
        const size_t smem = align16(acc_per_slot * ppc) + (smem_slots ? (size_t)ppc * slot_bytes : 0);
        const int64_t tiles = (a.chunk + ppc - 1) / ppc;
        void* kfn = smem_slots ? (void*)dpp_kernel<true> : (void*)dpp_kernel<false>;
        PT_CUDA(cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        int per_sm = 1;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kfn, threads, smem);
        per_sm = std::max(1, per_sm);
        const int grid = (int)std::max<int64_t>(1, std::min<int64_t>(tiles, (int64_t)ctx->num_sms * per_sm));
        const size_t bytes = align16(sizeof(DppPart) * (size_t)grid * nl) +
                             (smem_slots ? 0 : (size_t)grid * ppc * slot_bytes);
        void* scratch = nullptr;
        int rc = scratch_get(ctx, 1, bytes, &scratch);
        if (rc) return rc;
        DppLaunch L;
        L.mom = a.mom; L.chunk = a.chunk; L.nsave = a.nsave; L.lags = a.lags + lag0; L.nl = nl; L.p0 = a.p0;
        L.ppc = ppc; L.wps = wps; L.slot_bytes = slot_bytes;
        L.part = (DppPart*)scratch;
        L.gslots = smem_slots ? nullptr : (char*)scratch + align16(sizeof(DppPart) * (size_t)grid * nl);
        if (smem_slots) dpp_kernel<true><<<grid, threads, smem, s>>>(L);
        else dpp_kernel<false><<<grid, threads, smem, s>>>(L);
        PT_CHECK_LAUNCH("dpp_kernel");
        dpp_finalize_kernel<<<(nl + 255) / 256, 256, 0, s>>>(L.part, grid, nl, lag0, a.p0, a.counts, a.sdp, a.sdp2,
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
    if (smem > 48 * 1024)
        PT_CUDA(cudaFuncSetAttribute(energy_hist_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const double log_emin = log(e_min);
    const double inv_dlog = (double)n_hist / (log(e_max) - log_emin);
    const int blocks = (int)std::min<int64_t>((total + 255) / 256, 148 * 4);
    energy_hist_kernel<<<blocks, 256, smem, s>>>(mom, chunk, nsave, snaps, n_snap, log_emin, inv_dlog, n_hist,
                                                 (unsigned long long*)counts);
    PT_CHECK_LAUNCH("energy_hist_kernel");
    return PT_OK;
}

}  // namespace pt
