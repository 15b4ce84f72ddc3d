"""Parity of the CUDA lag statistics with the CPU oracle (needs a B200).

Bin counts and pair counts are compared bit for bit; FP64 sums and Welford
moments to 1e-12 relative (they differ only by summation order).  For the
signed sum of dmu the tolerance is relative to sqrt(count * sum dmu^2),
which bounds the sum of |dmu| the rounding acts on."""
import math

import numpy as np
import pytest

from helpers import random_mu_cache, zero_dmumu, zero_dpp
from particle_transport_b200 import stats as S
from particle_transport_b200.time_units import build_mu_edges_full, log_spaced_lag_steps

pytestmark = pytest.mark.gpu
RTOL = 1e-12


def close(a, b, rtol=RTOL, scale=None):
    a, b = np.asarray(a, float), np.asarray(b, float)
    tol = rtol * (np.abs(b) if scale is None else np.maximum(np.abs(b), scale)) + 1e-300
    return np.all(np.abs(a - b) <= tol)


def gpu_dmumu(mu, lags, edges, start_mode="sliding", bin_abs=True, layout="time_fastest", acc=None):
    nl, nb = len(lags), len(edges) - 1
    acc = acc or S.new_dmumu_accumulators(nl, nb)
    S.process_mu_chunk_dmumu(mu, lags, edges, acc["particle_counts"], acc["particle_means"], acc["particle_m2s"],
                             acc["pair_sum_squares"], acc["pair_counts"], acc["dmumu_counts"], acc["dmumu_sum_delta"],
                             acc["dmumu_sum_delta2"], start_mode=start_mode, bin_abs=bin_abs, layout=layout)
    return acc


def check_dmumu(g, o):
    assert np.array_equal(g["dmumu_counts"], o["counts"])
    assert np.array_equal(g["pair_counts"], o["pair_n"])
    assert np.array_equal(g["particle_counts"], o["w_count"])
    assert close(g["dmumu_sum_delta2"], o["sum_d2"])
    scale = np.sqrt(np.maximum(o["counts"], 1) * o["sum_d2"]) + 1e-30
    assert close(g["dmumu_sum_delta"], o["sum_d"], scale=scale)
    assert close(g["pair_sum_squares"], o["pair_ss"])
    assert close(g["particle_means"], o["w_mean"], rtol=1e-11)
    assert close(g["particle_m2s"], o["w_m2"], rtol=1e-9, scale=1e-300 + np.abs(o["w_m2"]).max() * 1e-3)


CASES = [
    # n, nsave, n_lags, n_bins, bin_abs, nan_frac, mode
    (4096, 801, 20, 20, True, 0.0, "sliding"),
    (333, 257, 40, 24, True, 0.05, "sliding"),
    (100, 120, 7, 10, False, 0.1, "sliding"),
    (1000, 401, 64, 50, True, 0.0, "injection"),
    (50, 64, 33, 5, False, 0.0, "injection"),
    (64, 300, 300, 8, True, 0.0, "sliding"),   # > 256 lags: several lag batches
    (3, 40001, 12, 16, True, 0.01, "sliding"),  # long series: staged in global memory
]


@pytest.mark.parametrize("n,nsave,n_lags,n_bins,bin_abs,nan_frac,mode", CASES)
def test_dmumu_matches_oracle(cuda, oracle, n, nsave, n_lags, n_bins, bin_abs, nan_frac, mode):
    mu = random_mu_cache(n, nsave, seed=n + nsave, nan_frac=nan_frac)
    lags = log_spaced_lag_steps(nsave - 1, n_lags) if n_lags < nsave else np.arange(1, n_lags + 1)
    edges, _ = build_mu_edges_full(0.0, 1.0, n_bins, bin_abs=bin_abs)
    o = zero_dmumu(len(lags), n_bins)
    oracle.dmumu_accumulate(mu, lags, edges, o, injection=mode == "injection", bin_abs=bin_abs)
    g = gpu_dmumu(mu, lags, edges, start_mode=mode, bin_abs=bin_abs)
    check_dmumu(g, o)


@pytest.mark.parametrize("bin_abs", [True, False])
def test_dmumu_non_uniform_edges(cuda, oracle, bin_abs):
    """Edges that are not a uniform range (the bin lookup starts from a
    uniform guess and walks to the stored edges), with values on the edges."""
    lo = 0.0 if bin_abs else -1.0
    edges = lo + (1.0 - lo) * np.linspace(0.0, 1.0, 18) ** 2
    rng = np.random.default_rng(11)
    mu = random_mu_cache(700, 301, seed=5, nan_frac=0.02)
    on_edge = rng.random(mu.shape) < 0.05
    mu[on_edge] = rng.choice(edges.astype(np.float32), size=int(on_edge.sum()))
    lags = log_spaced_lag_steps(300, 16)
    o = zero_dmumu(len(lags), 17)
    oracle.dmumu_accumulate(mu, lags, edges, o, bin_abs=bin_abs)
    check_dmumu(gpu_dmumu(mu, lags, edges, bin_abs=bin_abs), o)


def test_dmumu_chunks_add_into(cuda, oracle):
    """Two chunks accumulated into the same arrays == one oracle pass."""
    mu = random_mu_cache(900, 200, seed=4, nan_frac=0.02)
    lags = log_spaced_lag_steps(199, 16)
    edges, _ = build_mu_edges_full(0.0, 1.0, 12)
    o = zero_dmumu(len(lags), 12)
    oracle.dmumu_accumulate(mu, lags, edges, o)
    acc = gpu_dmumu(np.ascontiguousarray(mu[:317]), lags, edges)
    acc = gpu_dmumu(np.ascontiguousarray(mu[317:]), lags, edges, acc=acc)
    check_dmumu(acc, o)


def test_dmumu_device_particle_fastest(cuda, oracle):
    torch = cuda
    mu = random_mu_cache(2000, 161, seed=8, nan_frac=0.01)
    lags = log_spaced_lag_steps(160, 20)
    edges, _ = build_mu_edges_full(0.0, 1.0, 20)
    o = zero_dmumu(len(lags), 20)
    oracle.dmumu_accumulate(mu, lags, edges, o)
    d_mu = torch.as_tensor(np.ascontiguousarray(mu.T), device="cuda")  # [nsave][n]: the cache as written
    acc = S.new_dmumu_accumulators(len(lags), 20, device="cuda")
    gpu_dmumu(d_mu, lags, edges, layout="particle_fastest", acc=acc)
    torch.cuda.synchronize()
    check_dmumu({k: v.cpu().numpy() for k, v in acc.items()}, o)


def test_dmumu_edge_values(cuda, oracle):
    """Values on edges, |mu| = 1, signed out-of-range, NaN and Inf."""
    vals = np.array([0.0, 0.05, 0.1, 1.0, -1.0, 0.5, np.nan, np.inf, -np.inf, 0.95, 0.999999, 1e-30], np.float32)
    rng = np.random.default_rng(3)
    mu = np.ascontiguousarray(rng.choice(vals, size=(97, 130)).astype(np.float32))
    lags = np.array([1, 2, 3, 64, 129, 130, 500])
    for bin_abs in (True, False):
        edges, _ = build_mu_edges_full(0.0, 1.0, 20, bin_abs=bin_abs)
        o = zero_dmumu(len(lags), 20)
        oracle.dmumu_accumulate(mu, lags, edges, o, bin_abs=bin_abs)
        check_dmumu(gpu_dmumu(mu, lags, edges, bin_abs=bin_abs), o)


@pytest.mark.parametrize("mode", ["sliding", "injection"])
@pytest.mark.parametrize("edges", [[-np.inf, -0.5, 0.0, 0.5, np.inf], [-np.inf, 0.25], [-1.0, 0.0, np.inf]])
def test_dmumu_infinite_edges(cuda, oracle, mode, edges):
    """Signed bins open to one or both sides: finite values of any size have a bin, NaN and the infinities have
    none."""
    vals = np.array([0.0, -0.5, 0.25, 1.0, -1.0, 3e3, -3e3, np.nan, np.inf, -np.inf], np.float32)
    edges = np.array(edges)
    mu = np.ascontiguousarray(np.random.default_rng(4).choice(vals[[0, 1, 2, 3, 4, 7, 8, 9]], size=(97, 130)))
    mu[:, 0] = np.resize(vals, 97)  # the injection estimator's starts
    lags = np.array([1, 2, 64, 129, 500])
    o = zero_dmumu(len(lags), len(edges) - 1)
    oracle.dmumu_accumulate(mu, lags, edges, o, injection=mode == "injection", bin_abs=False)
    assert all(np.isfinite(o[k]).all() for k in ("sum_d", "sum_d2", "w_mean"))
    check_dmumu(gpu_dmumu(mu, lags, edges, start_mode=mode, bin_abs=False), o)


def test_dmumu_rejects_bad_lags(cuda):
    from particle_transport_b200._lib import PtError
    mu = random_mu_cache(4, 10)
    edges, _ = build_mu_edges_full(0.0, 1.0, 4)
    with pytest.raises(PtError, match="lag"):
        gpu_dmumu(mu, np.array([0, 1]), edges)


@pytest.mark.parametrize("chunk,nsave,n_lags", [(500, 201, 24), (37, 1000, 40), (2, 30001, 5), (64, 1500, 300),
                                                 (16, 6000, 500)])
def test_dpp_matches_oracle(cuda, oracle, chunk, nsave, n_lags):
    rng = np.random.default_rng(chunk)
    p = 5.4e-19 * (1 + 1e-3 * np.cumsum(rng.normal(size=(nsave, 1, chunk)), axis=0))
    u = rng.normal(size=(nsave, 3, chunk))
    u /= np.linalg.norm(u, axis=1, keepdims=True)
    mom = np.ascontiguousarray((p * u).astype(np.float32))
    mom[rng.random(mom.shape) < 0.001] = np.nan
    lags = log_spaced_lag_steps(nsave - 1, n_lags)
    p0 = 5.4e-19
    o = zero_dpp(len(lags))
    oracle.dpp_accumulate(mom, lags, p0, o)
    g = S.new_dpp_accumulators(len(lags))
    S.process_momenta_chunk_dpp(mom, lags, p0, g["counts"], g["sum_delta_p"], g["sum_delta_p2"],
                                g["sum_delta_p_norm"], g["sum_delta_p_norm2"])
    assert np.array_equal(g["counts"], o["counts"])
    assert close(g["sum_delta_p2"], o["sum_dp2"])
    assert close(g["sum_delta_p_norm2"], o["sum_dpn2"])
    sc = np.sqrt(np.maximum(o["counts"], 1) * o["sum_dp2"])
    assert close(g["sum_delta_p"], o["sum_dp"], scale=sc)
    sc = np.sqrt(np.maximum(o["counts"], 1) * o["sum_dpn2"])
    assert close(g["sum_delta_p_norm"], o["sum_dpn"], scale=sc)


def test_energy_snapshots_bit_exact(cuda, oracle):
    rng = np.random.default_rng(0)
    mom = np.ascontiguousarray(rng.normal(scale=5e-19, size=(50, 3, 300)).astype(np.float32))
    mom[3, :, 7] = np.nan
    snaps = np.array([0, 3, 25, 49])
    o = np.full((600, 4), np.nan)
    oracle.energy_snapshots(mom, snaps, o, particle_offset=300)
    g = np.full((600, 4), np.nan)
    S.fill_energy_snapshots(g, mom, snaps, particle_offset=300)
    assert np.array_equal(g, o, equal_nan=True)


def test_energy_snapshots_device_bit_exact(cuda, oracle):
    torch = cuda
    rng = np.random.default_rng(0)
    mom = np.ascontiguousarray(rng.normal(scale=5e-19, size=(50, 3, 300)).astype(np.float32))
    mom[3, :, 7] = np.nan
    snaps = np.array([0, 3, 25, 49])
    o = np.full((600, 4), np.nan)
    oracle.energy_snapshots(mom, snaps, o, particle_offset=300)
    g = torch.full((600, 4), float("nan"), dtype=torch.float64, device="cuda")
    S.fill_energy_snapshots(g, torch.as_tensor(mom, device="cuda"), snaps, particle_offset=300)
    assert np.array_equal(g.cpu().numpy(), o, equal_nan=True)
    # an index outside the chunk's saves yields NaN, not a stray read
    g2 = torch.zeros((300, 2), dtype=torch.float64, device="cuda")
    S.fill_energy_snapshots(g2, torch.as_tensor(mom, device="cuda"), [1, 50])
    h = g2.cpu().numpy()
    o1 = np.full((300, 1), np.nan)
    oracle.energy_snapshots(mom, np.array([1]), o1)
    assert np.all(np.isnan(h[:, 1])) and np.array_equal(h[:, 0], o1[:, 0], equal_nan=True)


def test_energy_histogram(cuda, oracle):
    torch = cuda
    rng = np.random.default_rng(1)
    mom = np.ascontiguousarray(rng.normal(scale=5e-18, size=(20, 3, 5000)).astype(np.float32))
    snaps = np.array([0, 10, 19])
    e = np.full((5000, 3), np.nan)
    oracle.energy_snapshots(mom, snaps, e)
    counts = S.energy_histogram(torch.as_tensor(mom, device="cuda"), snaps, 0.01, 100.0, 256).cpu().numpy()
    for j in range(3):
        ref, _ = np.histogram(e[:, j], bins=np.exp(np.linspace(math.log(0.01), math.log(100.0), 257)))
        assert counts[j].sum() == ref.sum()
        assert np.abs(counts[j] - ref).sum() <= 4  # log rounding at bin edges


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_reconstruct_mu_bit_exact(cuda, oracle, dtype):
    from helpers import copy_state, fortran_fields, small_problem
    pb = small_problem(n=12, n_particles=211)
    st = copy_state(pb.state)
    (pos, mom), _ = oracle.push_run(fortran_fields(pb.fields), pb.grid, st, np.ones(211, np.uint8), pb.dt, 120, 3,
                                    cache_mode=2, out_f64=dtype == np.float64)
    pos[5, 0, 3] = np.nan
    pos[6, 1, 4] = pb.grid.ymax * 1.01  # outside the box -> NaN
    ff = fortran_fields(pb.fields)[:3]
    if dtype == np.float64:
        o = oracle.reconstruct_mu_f64(pos, mom, ff, pb.grid)
    else:
        o = oracle.reconstruct_mu_f32(pos, mom, ff, pb.grid)
    g = S.reconstruct_mu_chunk(pos, mom, *pb.fields[:3], pb.grid, dtype=dtype)
    assert np.array_equal(g, o, equal_nan=True)
    assert np.isnan(g[3, 5]) and np.isnan(g[4, 6])


@pytest.mark.parametrize("b_layout", ["cells", "nodes"])
@pytest.mark.parametrize("dtype,mode,layout", [(np.float32, "sliding", "julia"), (np.float32, "injection", "cache"),
                                               (np.float64, "sliding", "cache")])
def test_phase_space_dmumu_fused_matches_oracle(cuda, oracle, dtype, mode, layout, b_layout, monkeypatch):
    """Fused phase-space D_mumu = oracle reconstruct_mu at the compute
    precision, then the oracle binning of that mu chunk -- with B read from
    8-corner cell records and from node records."""
    torch = cuda
    monkeypatch.setenv("PTB200_PHASE_SPACE_B", b_layout)
    from helpers import copy_state, fortran_fields, small_problem
    pb = small_problem(n=12, n_particles=517)
    st = copy_state(pb.state)
    f64 = dtype == np.float64
    (pos, mom), _ = oracle.push_run(fortran_fields(pb.fields), pb.grid, st, np.ones(517, np.uint8), pb.dt, 600, 3,
                                    cache_mode=2, out_f64=f64)
    pos[5, 0, 3] = np.nan
    pos[6, 1, 4] = pb.grid.ymax * 1.01  # outside the box -> NaN mu
    ff = fortran_fields(pb.fields)[:3]
    mu = (oracle.reconstruct_mu_f64 if f64 else oracle.reconstruct_mu_f32)(pos, mom, ff, pb.grid)  # (chunk, nsave)
    nsave = pos.shape[0]
    lags = log_spaced_lag_steps(nsave - 1, 24)
    edges, _ = build_mu_edges_full(0.0, 1.0, 16)
    o = zero_dmumu(len(lags), 16)
    # the reference bins Float64(mu) of the chunk at the compute precision; a Float32 chunk is exactly the oracle's input
    oracle.dmumu_accumulate(np.ascontiguousarray(mu, dtype=np.float32) if not f64 else mu, lags, edges, o,
                            injection=mode == "injection")
    tdt = torch.float64 if f64 else torch.float32
    if layout == "julia":
        P = torch.as_tensor(pos, dtype=tdt, device="cuda")
        M = torch.as_tensor(mom, dtype=tdt, device="cuda")
    else:  # the device phase-space cache (nsave, 6, n)
        cache = torch.cat([torch.as_tensor(pos, dtype=tdt), torch.as_tensor(mom, dtype=tdt)], dim=1).cuda()
        P, M = cache[:, 0:3], cache[:, 3:6]
    B = [torch.as_tensor(f, dtype=tdt, device="cuda") for f in pb.fields[:3]]
    g = S.new_dmumu_accumulators(len(lags), 16, device="cuda")
    S.process_phase_space_chunk_dmumu(P, M, *B, pb.grid, lags, edges, g["particle_counts"], g["particle_means"],
                                      g["particle_m2s"], g["pair_sum_squares"], g["pair_counts"], g["dmumu_counts"],
                                      g["dmumu_sum_delta"], g["dmumu_sum_delta2"], start_mode=mode)
    g = {k: v.cpu().numpy() for k, v in g.items()}
    check_dmumu(g, o)
    assert g["pair_counts"].sum() > 0


def _nan_pattern(mu, pattern, rng):
    """none; dead: NaN from some save on (open boundary); holes: NaN and Inf between finite saves; mixed."""
    n, nsave = mu.shape
    if pattern in ("dead", "mixed"):
        at = rng.integers(0, nsave + 1, size=n)  # 0: never alive, nsave: never dead
        sel = np.arange(n) % 2 == 0
        mu[(np.arange(nsave)[None, :] >= at[:, None]) & sel[:, None]] = np.nan
    if pattern in ("holes", "mixed"):
        m = rng.random(mu.shape)
        m[np.arange(n) % 3 == 0] = 1.0
        mu[m < 0.03] = np.nan
        mu[(m >= 0.03) & (m < 0.04)] = np.inf
    return mu


# the edges of the D_mumu launch shapes: one to eight lag sets of 8, then several lag groups and lag batches; one
# particle to more than a round; series stored four times on chip, once on chip (12,000 saves), and in global memory
# (30,000); injection tiles of 128 particles with a remainder, and lags beyond one warp
@pytest.mark.parametrize("n,nsave,n_lags,n_bins,mode,layout,pattern", [
    (1, 2, 1, 1, "sliding", "time_fastest", "none"),
    (37, 33, 8, 4, "sliding", "particle_fastest", "dead"),
    (700, 129, 9, 20, "sliding", "time_fastest", "mixed"),
    (150, 4001, 64, 50, "sliding", "time_fastest", "dead"),
    (301, 513, 41, 7, "sliding", "particle_fastest", "holes"),
    (90, 700, 65, 24, "sliding", "time_fastest", "mixed"),
    (64, 900, 130, 40, "sliding", "time_fastest", "dead"),
    (20, 12000, 30, 16, "sliding", "time_fastest", "mixed"),
    (5, 30000, 17, 40, "sliding", "particle_fastest", "mixed"),
    (40, 260, 32, 290, "sliding", "time_fastest", "none"),
    (1, 40, 5, 6, "injection", "time_fastest", "none"),
    (129, 300, 33, 20, "injection", "particle_fastest", "mixed"),
    (1000, 801, 64, 50, "injection", "time_fastest", "mixed"),
    (5000, 97, 7, 10, "injection", "particle_fastest", "dead"),
])
def test_dmumu_shapes_and_nan_patterns(cuda, oracle, n, nsave, n_lags, n_bins, mode, layout, pattern):
    """Counts bit for bit and sums to 1e-12 (as above) at the edges of the launch shapes, with lags past the series
    and values outside the edges; the tolerance is the summation-order bound of the other cases."""
    torch = cuda
    rng = np.random.default_rng(n + nsave + n_lags)
    mu = _nan_pattern(random_mu_cache(n, nsave, seed=nsave), pattern, rng)
    lags = np.concatenate([log_spaced_lag_steps(nsave - 1, n_lags) if n_lags < nsave else np.arange(1, n_lags + 1),
                           [nsave, 3 * nsave]])
    rng.shuffle(lags)
    edges = np.linspace(0.05, 0.9, n_bins + 1)
    o = zero_dmumu(len(lags), n_bins)
    oracle.dmumu_accumulate(mu, lags, edges, o, injection=mode == "injection", bin_abs=True)
    d = torch.as_tensor(mu if layout == "time_fastest" else np.ascontiguousarray(mu.T), device="cuda")
    acc = S.new_dmumu_accumulators(len(lags), n_bins, device="cuda")
    gpu_dmumu(d, lags, edges, start_mode=mode, layout=layout, acc=acc)
    check_dmumu({k: v.cpu().numpy() for k, v in acc.items()}, o)


# the edges of the D_pp launch shapes: one lag to more than 16 sets of 4, series counts of a CTA with a remainder, a
# last |p| chunk with fewer tiles than CTAs (2400 x 6000 saves), one series per CTA (13,000 saves), one CTA per SM
# (20,000), series in global memory (30,000)
@pytest.mark.parametrize("chunk,nsave,n_lags,pattern", [
    (1, 2, 1, "none"), (33, 65, 3, "dead"), (1000, 257, 16, "mixed"), (7, 300, 17, "holes"), (501, 402, 65, "dead"),
    (2400, 6000, 12, "mixed"), (40, 13000, 20, "dead"), (9, 20000, 9, "mixed"), (3, 30000, 66, "dead"),
])
def test_dpp_shapes_and_nan_patterns(cuda, oracle, chunk, nsave, n_lags, pattern):
    """As test_dpp_matches_oracle (counts exact, sums to 1e-12 of the sums the rounding acts on), on the device entry,
    with particles that die and NaN or Inf between finite saves, and lags past the series."""
    torch = cuda
    rng = np.random.default_rng(chunk + nsave)
    p = 5.4e-19 * (1 + 1e-3 * np.cumsum(rng.normal(size=(nsave, 1, chunk)), axis=0))
    u = rng.normal(size=(nsave, 3, chunk))
    u /= np.linalg.norm(u, axis=1, keepdims=True)
    mom = (p * u).astype(np.float32)
    hide = _nan_pattern(np.zeros((chunk, nsave), np.float32), pattern, rng).T
    mom[:, 1] = np.where(np.isfinite(hide), mom[:, 1], hide)
    mom = np.ascontiguousarray(mom)
    lags = np.concatenate([log_spaced_lag_steps(nsave - 1, n_lags), [nsave, 2 * nsave]])
    rng.shuffle(lags)
    p0 = 5.4e-19
    o = zero_dpp(len(lags))
    oracle.dpp_accumulate(mom, lags, p0, o)
    acc = S.new_dpp_accumulators(len(lags), device="cuda")
    S.process_momenta_chunk_dpp(torch.as_tensor(mom, device="cuda"), lags, p0, acc["counts"], acc["sum_delta_p"],
                                acc["sum_delta_p2"], acc["sum_delta_p_norm"], acc["sum_delta_p_norm2"])
    g = {k: v.cpu().numpy() for k, v in acc.items()}
    assert np.array_equal(g["counts"], o["counts"])
    assert close(g["sum_delta_p2"], o["sum_dp2"])
    assert close(g["sum_delta_p_norm2"], o["sum_dpn2"])
    assert close(g["sum_delta_p"], o["sum_dp"], scale=np.sqrt(np.maximum(o["counts"], 1) * o["sum_dp2"]))
    assert close(g["sum_delta_p_norm"], o["sum_dpn"], scale=np.sqrt(np.maximum(o["counts"], 1) * o["sum_dpn2"]))


# B read as the arrays are (few samples per node), as cell and as node records; tiles of 32 particles with a remainder;
# the injection estimator's saves alone, with lags past the series
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("mode", ["sliding", "injection"])
@pytest.mark.parametrize("b_layout", [None, "cells", "nodes"])
def test_phase_space_dmumu_b_sources(cuda, oracle, dtype, mode, b_layout, monkeypatch):
    """As test_phase_space_dmumu_fused_matches_oracle on a grid with more nodes than samples."""
    torch = cuda
    monkeypatch.delenv("PTB200_PHASE_SPACE_B", raising=False)
    if b_layout:
        monkeypatch.setenv("PTB200_PHASE_SPACE_B", b_layout)
    from helpers import copy_state, fortran_fields, small_problem
    pb = small_problem(n=40, n_particles=70)
    f64 = dtype == np.float64
    (pos, mom), _ = oracle.push_run(fortran_fields(pb.fields), pb.grid, copy_state(pb.state), np.ones(70, np.uint8),
                                    pb.dt, 292, 3, cache_mode=2, out_f64=f64)
    pos[7, 0, 3] = np.nan
    pos[60:, 1, 4] = np.nan  # a particle that died
    pos[0, 2, 69] = pb.grid.zmax * 1.01  # outside the box at the first save
    ff = fortran_fields(pb.fields)[:3]
    mu = (oracle.reconstruct_mu_f64 if f64 else oracle.reconstruct_mu_f32)(pos, mom, ff, pb.grid)
    nsave = pos.shape[0]
    lags = np.concatenate([log_spaced_lag_steps(nsave - 1, 40), [nsave, 5 * nsave]])
    edges, _ = build_mu_edges_full(0.0, 1.0, 16)
    o = zero_dmumu(len(lags), 16)
    oracle.dmumu_accumulate(mu, lags, edges, o, injection=mode == "injection")
    tdt = torch.float64 if f64 else torch.float32
    P, M = (torch.as_tensor(v, dtype=tdt, device="cuda") for v in (pos, mom))
    B = [torch.as_tensor(f, dtype=tdt, device="cuda") for f in pb.fields[:3]]
    g = S.new_dmumu_accumulators(len(lags), 16, device="cuda")
    S.process_phase_space_chunk_dmumu(P, M, *B, pb.grid, lags, edges, g["particle_counts"], g["particle_means"],
                                      g["particle_m2s"], g["pair_sum_squares"], g["pair_counts"], g["dmumu_counts"],
                                      g["dmumu_sum_delta"], g["dmumu_sum_delta2"], start_mode=mode)
    check_dmumu({k: v.cpu().numpy() for k, v in g.items()}, o)


@pytest.mark.parametrize("kind", ["dmumu", "dpp"])
def test_longest_series(cuda, kind):
    """One particle with the most saves that the entries take, 2^31 - 2: loops over saves and starts end where the
    series does.  The values are multiples of a power of two, so that every sum is exact."""
    torch = cuda
    ns = 2**31 - 2
    if torch.cuda.mem_get_info()[0] < 80 << 30:
        pytest.skip("needs 80 GB of device memory")
    lags = np.array([1, ns - 1, 7, ns - 3])
    if kind == "dmumu":
        vals = np.array([0.125, 0.25, 0.5, 0.75, 0.875])
        mu = torch.as_tensor(vals, dtype=torch.float32, device="cuda").repeat(ns // 5 + 1)[:ns].view(1, ns)
        acc = S.new_dmumu_accumulators(len(lags), 5, device="cuda")
        gpu_dmumu(mu, lags, np.linspace(0.0, 1.0, 6), acc=acc)
        g = {k: v.cpu().numpy() for k, v in acc.items()}
        del mu
        for i, L in enumerate(lags):
            c = (ns - L - np.arange(5) + 4) // 5  # starts of each value that reach the lag
            d = np.roll(vals, -(L % 5)) - vals
            assert np.array_equal(g["dmumu_counts"][i], c)
            assert np.array_equal(g["dmumu_sum_delta"][i], c * d)
            assert np.array_equal(g["dmumu_sum_delta2"][i], c * d * d)
            assert g["pair_counts"][i] == ns - L and g["particle_counts"][i] == 1
            assert g["particle_means"][i] == (c * d * d).sum() / (ns - L)
    else:
        vals = np.array([1.0, 2.0, 4.0]) * 2.0**-63
        mom = torch.zeros((ns, 3, 1), dtype=torch.float32, device="cuda")
        mom[:, 1, 0] = torch.as_tensor(vals, dtype=torch.float32, device="cuda").repeat(ns // 3)
        acc = S.new_dpp_accumulators(len(lags), device="cuda")
        S.process_momenta_chunk_dpp(mom, lags, 1.0, acc["counts"], acc["sum_delta_p"], acc["sum_delta_p2"],
                                    acc["sum_delta_p_norm"], acc["sum_delta_p_norm2"])
        g = {k: v.cpu().numpy() for k, v in acc.items()}
        del mom
        for i, L in enumerate(lags):
            c = (ns - L - np.arange(3) + 2) // 3
            d = np.roll(vals, -(L % 3)) - vals
            assert g["counts"][i] == ns - L
            assert g["sum_delta_p"][i] == (c * d).sum() and g["sum_delta_p2"][i] == (c * d * d).sum()
    torch.cuda.empty_cache()


def test_calls_of_several_threads(cuda):
    """Threads, each with its own context, make calls of the same kernels that need different amounts of shared
    memory: every call launches, and the sums are those of the calls alone."""
    torch = cuda
    import threading
    from particle_transport_b200 import _lib
    lags = torch.as_tensor(np.array([1, 2, 5, 9, 17, 30]), device="cuda")
    edges = torch.linspace(0.0, 1.0, 11, dtype=torch.float64, device="cuda")
    ins = [(torch.as_tensor(random_mu_cache(20, ns, seed=ns), device="cuda"), torch.ones((ns, 3, 4), device="cuda"))
           for ns in (64, 3001, 11000)]

    def calls(ctx, mu, mom, reps):
        a, b = S.new_dmumu_accumulators(6, 10, device="cuda"), S.new_dpp_accumulators(6, device="cuda")
        keys = ("dmumu_counts", "dmumu_sum_delta", "dmumu_sum_delta2", "particle_counts", "particle_means",
                "particle_m2s", "pair_sum_squares", "pair_counts")
        args = [_lib.ptr(mu), *mu.shape, mu.shape[1], 1, _lib.ptr(lags), 6, _lib.ptr(edges), 10, 0, 1,
                *[_lib.ptr(a[k]) for k in keys]]
        dpp = [_lib.ptr(mom), 4, mu.shape[1], _lib.ptr(lags), 6, 1.0,
               *[_lib.ptr(b[k]) for k in ("counts", "sum_delta_p", "sum_delta_p2", "sum_delta_p_norm",
                                          "sum_delta_p_norm2")]]
        torch.cuda.synchronize()
        for _ in range(reps):
            _lib.call("pt_dmumu_accumulate_device", ctx.handle, *args)
            _lib.call("pt_dpp_accumulate_device", ctx.handle, *dpp)
        ctx.synchronize()
        return torch.cat([a["dmumu_counts"].flatten(), a["pair_counts"], b["counts"]])

    ctxs = [_lib.Context(0) for _ in ins]
    want = [calls(c, *i, 1) for c, i in zip(ctxs, ins)]
    got, errors = [None] * len(ins), []

    def work(i):
        try:
            got[i] = calls(ctxs[i], *ins[i], 3000)
        except Exception as e:
            errors.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(ins))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]
    for g, w in zip(got, want):
        assert torch.equal(g, 3000 * w)
    for c in ctxs:
        c.close()


def test_dpp_on_a_full_device(cuda):
    """D_pp with less free memory than its |p| chunks would take, and inside a stream capture: the same sums from
    smaller chunks."""
    torch = cuda
    from particle_transport_b200 import _lib
    n, ns = 20000, 1001
    g = torch.Generator(device="cuda").manual_seed(5)
    mom = torch.randn((ns, 3, n), generator=g, device="cuda")
    mom[500:, :, ::3] = float("nan")
    lags = torch.as_tensor(log_spaced_lag_steps(ns - 1, 12), device="cuda")
    nl = len(lags)
    keys = ("counts", "sum_delta_p", "sum_delta_p2", "sum_delta_p_norm", "sum_delta_p_norm2")
    accs = [S.new_dpp_accumulators(nl, device="cuda") for _ in range(3)]

    def call(ctx, acc, m=n):
        _lib.call("pt_dpp_accumulate_device", ctx.handle, _lib.ptr(mom), m, ns, _lib.ptr(lags), nl, 2.0,
                  *[_lib.ptr(acc[k]) for k in keys])

    call(_lib.torch_context(0), accs[0])
    ctx = _lib.Context(0)
    ctx.use_stream(torch.cuda.current_stream())
    call(ctx, S.new_dpp_accumulators(nl, device="cuda"), 7)  # what the context keeps between calls is there
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    held = []
    while torch.cuda.mem_get_info()[0] > 96 << 20:
        held.append(torch.empty(torch.cuda.mem_get_info()[0] - (64 << 20), dtype=torch.uint8, device="cuda"))
    call(ctx, accs[1])
    torch.cuda.synchronize()
    del held
    torch.cuda.empty_cache()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        ctx.use_stream(torch.cuda.current_stream())
        call(ctx, accs[2])
    graph.replay()
    torch.cuda.synchronize()
    ctx.use_stream(None)
    want = {k: v.cpu().numpy() for k, v in accs[0].items()}
    for acc in accs[1:]:
        got = {k: v.cpu().numpy() for k, v in acc.items()}
        assert np.array_equal(got["counts"], want["counts"])
        assert close(got["sum_delta_p2"], want["sum_delta_p2"]) and close(got["sum_delta_p_norm2"],
                                                                         want["sum_delta_p_norm2"])
        scale = np.sqrt(np.maximum(want["counts"], 1) * want["sum_delta_p2"])
        assert close(got["sum_delta_p"], want["sum_delta_p"], scale=scale)
        assert close(got["sum_delta_p_norm"], want["sum_delta_p_norm"], scale=scale)
    del graph
    ctx.close()


# 1, 2, 4 and 8 lag sets, whose 16, 8, 4 and 2 warps share the particles of a tile or the starts of a series; series
# shorter than a warp (several in one warp's copies), tiles with a remainder, an even and an odd number of saves
@pytest.mark.parametrize("chunk,nsave,n_lags,pattern", [
    (4801, 9, 1, "mixed"), (5000, 40, 2, "mixed"), (4999, 201, 5, "holes"), (700, 3000, 2, "dead"),
    (2999, 900, 14, "mixed"), (301, 4001, 27, "holes"), (2, 30001, 3, "mixed"), (4737, 64, 30, "none"),
])
def test_dpp_few_lags(cuda, oracle, chunk, nsave, n_lags, pattern):
    """As test_dpp_shapes_and_nan_patterns, where a set of lags has several warps."""
    test_dpp_shapes_and_nan_patterns(cuda, oracle, chunk, nsave, n_lags, pattern)
