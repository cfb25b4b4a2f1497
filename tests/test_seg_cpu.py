"""The arithmetic of the tiled assemblies (edge matrices of seg_device.cuh, side
matrices of hs_device.cuh), compiled for the host, against the oracle's tractions
(the published angular dislocations and free-surface correction in the reference's
operation order), with edges walked either way and two Poisson ratios.  Each pair
within 1e-10 of its largest traction, the project's parity bar, of the published
formula in long double -- and, where the oracle's own FP64 evaluation is further from
that (far receivers of thin triangles: up to 7e-10), no further than the oracle.  In
the half space the sides are at least 10 degrees off the vertical, where the published
formula itself keeps its digits."""
import os
import shutil
import subprocess

import numpy as np
import pytest

import oracle

MU = 32038120320.0
HERE = os.path.dirname(os.path.abspath(__file__))


def _build(tmp_path_factory, name):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.fail("no C++ compiler for the host build of the device math")
    exe = str(tmp_path_factory.mktemp("seg") / name)
    subprocess.run([cxx, "-O2", "-std=c++17", "-o", exe, os.path.join(HERE, name + ".cpp")], check=True)
    return exe


@pytest.fixture(scope="module")
def seg_check(tmp_path_factory):
    return _build(tmp_path_factory, "seg_host_check")


@pytest.fixture(scope="module")
def exact_check(tmp_path_factory):
    return _build(tmp_path_factory, "pair_exact_check")


def _frame(n):
    n = n / np.linalg.norm(n)
    e1 = np.cross([0.0, 0.0, 1.0], n)
    e1 /= np.linalg.norm(e1)
    return e1, np.cross(n, e1), n


def _tractions(P, X, F, lam, half):
    out = []
    for slip in ((1.0, 0.0), (0.0, 1.0)):
        s, _ = oracle.tdstress(X[:1].copy(), X[1:2].copy(), X[2:3].copy(), *P, *slip, 0.0, MU, lam, half)
        T = s[0][[0, 3, 4, 3, 1, 5, 4, 5, 2]].reshape(3, 3)
        out += [a @ T @ F[2] for a in F]
    return np.array(out)


def _run(exe, cases, ratio):
    inp = "%d %.17g\n" % (len(cases), ratio) + "\n".join(
        " ".join("%.17g" % v for v in np.concatenate([P.ravel(), X, *F])) + " %d" % r for P, X, F, r in cases)
    out = subprocess.run([exe], input=inp, capture_output=True, text=True, check=True).stdout
    return np.array([[float(v) for v in line.split()] for line in out.strip().split("\n")])


@pytest.mark.parametrize("ratio", [1.0, 0.6])
def test_full_space_pairs(seg_check, exact_check, ratio):
    rng = np.random.default_rng(11)
    cases = []
    for t in range(500):
        P = rng.normal(size=(3, 3)) * 2000 + np.array([0, 0, -8000.0])
        if t % 3 == 0:   # in the source's plane, inside and outside, off the side lines
            s, u = rng.uniform(-1.5, 2.5, size=2)
            X = P[0] + s * (P[1] - P[0]) + u * (P[2] - P[0])
        else:
            X = P.mean(axis=0) + rng.normal(size=3) * rng.choice([300.0, 3000.0, 30000.0, 300000.0])
        cases.append((P, X, _frame(rng.normal(size=3)), int(rng.integers(8))))
    for (P, X, F, _), got, exact in zip(cases, _run(seg_check, cases, ratio), _run(exact_check, cases, ratio)):
        ref = _tractions(P, X, F, ratio * MU, False)
        bar = max(1e-10 * np.abs(exact[:6]).max(), np.abs(ref - exact[:6]).max())
        assert np.abs(got[:6] - exact[:6]).max() <= bar


@pytest.mark.parametrize("ratio", [1.0, 0.6])
def test_half_space_pairs(seg_check, exact_check, ratio):
    rng = np.random.default_rng(12)
    cases = []
    while len(cases) < 400:
        P = rng.normal(size=(3, 3)) * 2000 + np.array([0, 0, -5000.0])
        P[:, 2] = -np.abs(P[:, 2])
        if len(cases) % 7 == 0:
            P[0, 2] = P[1, 2] = 0.0   # an edge in the surface
        sides = P[[1, 2, 0]] - P
        if (np.hypot(sides[:, 0], sides[:, 1]) < np.sin(np.radians(10.0)) * np.linalg.norm(sides, axis=1)).any():
            continue
        X = np.array([rng.uniform(-9000, 9000), rng.uniform(-9000, 9000), -rng.uniform(100.0, 10000)])
        cases.append((P, X, _frame(rng.normal(size=3)), int(rng.integers(8))))
    for (P, X, F, _), got, exact in zip(cases, _run(seg_check, cases, ratio), _run(exact_check, cases, ratio)):
        ref = _tractions(P, X, F, ratio * MU, True)
        bar = max(1e-10 * np.abs(exact).max(), np.abs(ref - exact[6:]).max())
        assert np.abs(got[6:] - exact[6:]).max() <= bar


def test_an_edge_walked_backwards_is_its_negative(seg_check):
    rng = np.random.default_rng(13)
    cases = []
    for _ in range(60):
        P = rng.normal(size=(3, 3)) * 2000 + np.array([0, 0, -9000.0])
        X = P.mean(axis=0) + rng.normal(size=3) * 4000.0
        X[2] = min(X[2], -50.0)
        F = _frame(rng.normal(size=3))
        cases += [(P, X, F, r) for r in range(8)]
    got = _run(seg_check, cases, 1.0).reshape(60, 8, 12)
    scale = np.abs(got).max(axis=(1, 2), keepdims=True)
    assert (np.abs(got - got[:, :1]) <= 1e-10 * scale).all()


def test_receivers_on_an_edge_are_marked(seg_check):
    """Within 1e-6 of an edge's length beside it: NaN, which the kernels take for
    the pair evaluation; beyond the edge's ends and off it: none."""
    P = np.array([[0.0, 0.0, -5000.0], [3000.0, 400.0, -5200.0], [700.0, 2500.0, -6400.0]])
    F = _frame(np.array([0.3, -0.5, 0.8]))
    d = P[1] - P[0]
    L = np.linalg.norm(d)
    off = np.cross(d, [0.0, 0.0, 1.0])
    off /= np.linalg.norm(off)
    xs = [P[0] + 0.37 * d + k * L * off for k in (0.0, 5e-7, 3e-6, 1e-2)] + [P[0] - 0.2 * d, P[0] + 1.3 * d, P[1]]
    got = _run(seg_check, [(P, x, F, 0) for x in xs], 1.0)
    assert [bool(np.isnan(g[:6]).any()) for g in got] == [True, True, False, False, False, False, True]
