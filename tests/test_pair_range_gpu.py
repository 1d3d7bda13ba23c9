"""FP64 pair sums and metric over wide ranges of the operands, marker by marker, against
sums in extended precision: coordinates far below the size of the domain, close pairs
near the origin, clusters of small G.

Bound: at most twice the error of the one-sided FP64 kernels on the same inputs. An error
is taken relative to the sizes of a marker's terms, w_a |G_a - G_g| / |d| (the metric:
w_a / |d|), and of all markers the largest counts; below two units of 2^-53 (the rounding
of the final sum) any error will do.
"""
from __future__ import annotations

import numpy as np
import pytest

from conftest import gaussian_markers

pytestmark = pytest.mark.gpu


def sums(v, w, G):
    """F, A and the sizes of their terms, in extended precision (N x 2, N x 3, N, N)."""
    L = np.longdouble
    v, w, G = v.astype(L), w.astype(L), G.astype(L)
    N = len(w)
    F, A, sf, sa = np.zeros((N, 2), L), np.zeros((N, 3), L), np.zeros(N, L), np.zeros(N, L)
    for i in range(0, N, 100):
        s = slice(i, i + 100)
        d1, d2 = v[s, None, 0] - v[:, 0], v[s, None, 1] - v[:, 1]
        g1, g2 = G[:, 0] - G[s, None, 0], G[:, 1] - G[s, None, 1]
        r2 = d1 * d1 + d2 * d2
        r = np.where(r2 < 1e-24, np.inf, np.sqrt(r2))
        k = w / (r * r * r)
        c = k * (g1 * d2 - g2 * d1)
        F[s] = np.stack([(c * d2).sum(1), -(c * d1).sum(1)], 1)
        A[s] = np.stack([(k * d2 * d2).sum(1), -(k * d1 * d2).sum(1), (k * d1 * d1).sum(1)], 1)
        sf[s] = (np.abs(w) * np.sqrt(g1 * g1 + g2 * g2) / r).sum(1)
        sa[s] = (np.abs(w) / r).sum(1)
    return F, A, sf, sa


def check(collops, bp, v, w, G):
    N = len(w)
    v, G = np.asfortranarray(v), np.asfortranarray(G)
    Fr, Ar, sf, sa = sums(v, w, G)
    err = {}
    for onesided in (True, False):
        ws = collops.build_workspace(
            collops.SimParameters(bp1=bp, bp2=bp, pair_onesided=onesided))
        dv, F, A = (np.zeros((N, k), order="F") for k in (2, 2, 3))
        collops.compute_collision_gpu(ws, dv, v, w, G)
        collops.compute_collision_metric_gpu(ws, F, A, v, w, G)
        ws.close()
        err[onesided] = [float(np.max(np.abs(got - ref) / size[:, None])) for got, ref, size in
                         ((dv, Fr, sf), (F, Fr, sf), (A, Ar, sa))]
    for here, fp64 in zip(err[False], err[True]):
        assert here <= max(2 * fp64, 2.0 ** -52)


def graded(half):
    return np.concatenate([np.linspace(-6.0, 6.0, 13)] if half == 6.0 else
                          [[-half], np.linspace(-6.0, 6.0, 13), [half]])


def _markers(N, seed, weights="random"):
    v, w = gaussian_markers(N, 1.0, 0.6, seed=seed)
    rng = np.random.default_rng(seed)
    if weights == "random":
        w = rng.uniform(0.2, 1.8, N) / N
    G = -v / [1.0, 0.36] + 0.2 * np.sin(2 * v[:, ::-1]) + 0.05 * rng.standard_normal(v.shape)
    return v, w, G


@pytest.mark.parametrize("weights", ["equal", "random"])
@pytest.mark.parametrize("half", [6.0, 1e2, 1e4, 1e6])
def test_wide_domains(built_lib, collops_mod, half, weights):
    """Markers of thermal width 1 in domains of larger and larger half-width."""
    check(collops_mod, graded(half), *_markers(1200, 3, weights))


@pytest.mark.parametrize("gap", [4.1e-6, 4e-5, 1e-3])
def test_close_pairs_near_the_origin(built_lib, collops_mod, gap):
    """Pairs beyond the reach of the FP64 form whose coordinates are all small."""
    v, w, G = _markers(1200, 5)
    rng = np.random.default_rng(8)
    v[:200] = 0.05 * (rng.random((200, 2)) - 0.5)
    t = rng.uniform(0, 2 * np.pi, 100)
    v[100:200] = v[:100] + gap * np.stack([np.cos(t), np.sin(t)], 1)
    check(collops_mod, graded(6.0), v, w, G)


@pytest.mark.parametrize("share", [2, 10])
@pytest.mark.parametrize("k", [6, 12, 18])
def test_cold_core(built_lib, collops_mod, k, share):
    """A share of the markers 2^k times colder than the rest, with a smooth G."""
    v, w, G = _markers(1200, 7)
    v[::share] *= 2.0 ** -k
    G[::share] *= 2.0 ** -k
    check(collops_mod, graded(6.0), v, w, G)


def test_sums_of_one_term(built_lib, collops_mod):
    """Each marker 0.005 to 0.02 from one of 32 weighted ones, the others weightless: its sum
    is next to one term, whose error nothing averages."""
    v, w, G = _markers(512, 27)
    rng = np.random.default_rng(28)
    w = np.where(np.arange(512) % 16 == 0, w, 0.0)
    t, d = rng.uniform(0, 2 * np.pi, 512), rng.uniform(0.005, 0.02, 512)
    at = 16 * rng.integers(0, 32, 512)
    near = v[at] + d[:, None] * np.stack([np.cos(t), np.sin(t)], 1)
    v = np.where(w[:, None] > 0.0, v, near)
    check(collops_mod, graded(6.0), v, w, rng.standard_normal((512, 2)))


@pytest.mark.parametrize("seed", range(4))
def test_light_close_pairs(built_lib, collops_mod, seed):
    """Pairs just beyond the reach of the FP64 form, of markers whose weights lie over eight
    decades: a light one's term is small, but not its 1/|d|."""
    v, w, G = _markers(400, 29 + seed)
    rng = np.random.default_rng(30 + seed)
    t = rng.uniform(0, 2 * np.pi, 200)
    gap = 10.0 ** rng.uniform(-5.2, -5, 200)
    v[200:] = v[:200] + gap[:, None] * np.stack([np.cos(t), np.sin(t)], 1)
    w *= 10.0 ** (-8 * rng.random(400))
    check(collops_mod, graded(6.0), v, w, G)


def test_tiny_domain(built_lib, collops_mod, oracle_mod):
    """A domain so small that the guard distance 1e-12 is far beyond the usual reach of the
    FP64 form. Against the CPU oracle: sums of N FP64 terms, ten times sqrt(N) 2^-53."""
    v, w, G = _markers(1200, 9)
    v = np.asfortranarray(v * 2.0 ** -38)
    G = np.asfortranarray(G)
    bp = graded(6.0) * 2.0 ** -38
    ws = collops_mod.build_workspace(collops_mod.SimParameters(bp1=bp, bp2=bp))
    F, A = np.zeros((1200, 2), order="F"), np.zeros((1200, 3), order="F")
    collops_mod.compute_collision_metric_gpu(ws, F, A, v, w, G)
    ws.close()
    Fr, Ar = oracle_mod.OracleMesh(bp, bp, 6).collision_metric(v, w, G)
    for got, ref in ((F, Fr), (A, Ar)):
        assert np.max(np.abs(got - ref)) <= 10 * 1200 ** 0.5 * 2.0 ** -53 * np.max(np.abs(ref))


@pytest.mark.parametrize("size", [1e2, 1e3, 1e5, 1e8, 1e12, 1e17])
@pytest.mark.parametrize("weight", [0.0, 1e-14])
def test_one_huge_gradient(built_lib, collops_mod, weight, size):
    """A marker of (next to) no weight with a G far above the others': it adds nothing to
    them and must not cost them digits."""
    v, w, G = _markers(1200, 11)
    w[400] *= weight
    G[400, 0] = size
    check(collops_mod, graded(6.0), v, w, G)


@pytest.mark.parametrize("ratio", [1e1, 1e2, 1e4, 1e12])
def test_one_heavy_marker(built_lib, collops_mod, ratio):
    v, w, G = _markers(1200, 13)
    w /= ratio
    w[700] = 1.0 / 1200
    check(collops_mod, graded(6.0), v, w, G)


@pytest.mark.parametrize("balanced", [False, True])
@pytest.mark.parametrize("decades", [2, 4, 12])
def test_weights_over_decades(built_lib, collops_mod, decades, balanced):
    """Weights log-uniform over decades, with G of one size or balanced, G ~ 1/w."""
    v, w, G = _markers(1200, 17)
    s = 10.0 ** (-decades * np.random.default_rng(4).random(1200))
    w *= s
    if balanced:
        G /= s[:, None]
    check(collops_mod, graded(6.0), v, w, G)


@pytest.mark.parametrize("offset", [1e2, 1e4, 1e8])
def test_common_part_of_the_gradient(built_lib, collops_mod, offset):
    """Only differences of G count."""
    v, w, G = _markers(1200, 19)
    check(collops_mod, graded(6.0), v, w, G + [offset, -0.3 * offset])


def test_map_of_unequal_weights(built_lib, collops_mod, oracle_mod):
    """The map forms lambda dv / w itself, so weights over twelve decades give a G over as
    many: a marker's error against the CPU oracle at most twice that of the one-sided FP64
    kernels, or one unit of 2^-52 of its velocity."""
    N = 1200
    v, w, _ = _markers(N, 23)
    w = w * 10.0 ** (-12 * np.random.default_rng(6).random(N))
    v = np.asfortranarray(v)
    v_in = np.asfortranarray(v - 0.01 * v + 0.001 * np.sin(3 * v[:, ::-1]))
    bp = np.linspace(-6.0, 6.0, 13)
    om = oracle_mod.OracleMesh(bp, bp, 6)
    S0 = om.entropy(om.l2_project(v, w))
    ref = om.picard_map(oracle_mod.Opts(), v_in, v, w, S0, 0.01)
    err = {}
    for onesided in (True, False):
        ws = collops_mod.build_workspace(
            collops_mod.SimParameters(bp1=bp, bp2=bp, pair_onesided=onesided))
        out = np.zeros((N, 2), order="F")
        collops_mod.picard_map(ws, out, v_in, v, w, S0, 0.01)
        ws.close()
        err[onesided] = float(np.max(np.linalg.norm(out - ref, axis=1) / np.linalg.norm(ref, axis=1)))
    assert err[False] <= max(2 * err[True], 2.0 ** -52)
