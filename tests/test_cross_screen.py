"""The per-event screen of the streaming forward kernels (may_cross with cross_window, bats_gb300/csrc/common.cuh)
is conservative: wherever it says that no crossing has to be looked for, no value of __expf and __logf within
their documented error bounds lets the reference solver accept one. The device source is compiled for the host
(as in tests/test_screen_source.py: the screen's comparisons hold no product-plus-sum that nvcc could fuse but
the explicit ones) and evaluated on states built with a root just outside the window, the edge of the proof.
The solver that it gates (solve_candidate) gives the reference loop's results bit for bit on 4 10^6 windows."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from tests import test_screen_source as screen_source
from tests import test_solver_source as solver_source
from tests._float_model import F, expf_range, reference_may_accept, states_with_root_near
from tests.test_event_screen import NO_T, TAUS, THETAS
from tests.test_screen_source import _cuda_include, _run, _wild

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# modes 0 (FC) and 1 (conv) answer with the new screen's claim instead of no_crossing's
SCREEN = screen_source.PROGRAM.replace("        bool r;\n", "        bats::set_screen_const(k);\n        bool r;\n").replace(
    "bats::no_crossing<false>(v[i], v[n + i], v[2 * n + i], v[3 * n + i], k);",
    "!bats::may_cross<false>(v[i], v[n + i], bats::cross_window(0, 0, v[2 * n + i], v[3 * n + i], k), k);").replace(
    "bats::no_crossing<true>(v[i], v[n + i], v[2 * n + i], v[3 * n + i], k);",
    "!bats::may_cross<true>(v[i], v[n + i], bats::cross_window(0, 0, v[2 * n + i], v[3 * n + i], k), k);")

SOLVER = solver_source.PROGRAM.replace("        k.fast = true;\n", "        k.fast = true;\n        bats::set_screen_const(k);\n").replace(
    "if (bats::no_crossing<CONV>(a, b, e_ev, e_nx, k)) ++screened;",
    "const bats::CrossWindow w = bats::cross_window(0, 0, e_ev, e_nx, k);\n"
    "        const bool look = bats::may_cross<CONV>(a, b, w, k);\n        screened += !look;").replace(
    "const bool r2 = bats::solve_crossings<CONV>(a, b2, t_ev, next, e_ev, e_nx, k, n2, K, ao2, xo2, to2, zo2);",
    "const bool r2 = look && bats::solve_candidate<CONV>(a, b2, t_ev, next, w, k, n2, K, 0, ao2, xo2, to2, zo2);")


def _build(tmp, name, text):
    inc = _cuda_include()
    if shutil.which("g++") is None or inc is None:
        pytest.skip("no host C++ compiler or CUDA headers")
    src, exe = tmp / (name + ".cpp"), tmp / name
    src.write_text(text)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", os.path.join(ROOT, "bats_gb300", "csrc"),
                    "-I", inc, "-o", str(exe), str(src)], check=True)
    return str(exe)


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    assert SCREEN.count("may_cross") == 2 and SCREEN.count("set_screen_const") == 1
    return _build(tmp_path_factory.mktemp("cross"), "screen", SCREEN)


def _claims(exe, conv, a, b, e_start, e_next, c, e_max):
    full = [np.broadcast_to(np.asarray(v, F), a.shape) for v in (a, b, e_start, e_next, c, e_max)]
    return _run(exe, int(conv), full)


@pytest.mark.parametrize("conv", [False, True], ids=["fc", "conv"])
def test_claims_at_the_windows_end_are_never_accepted(exe, conv):
    """Smaller root within a few 2^-20 of the next event (also near 8 tau) or of max_sim. Planted: the screen is
    given a window that ends 2^-14 early."""
    rng = np.random.default_rng(21)
    claims = planted = 0
    for tau in TAUS:
        for theta in THETAS:
            c, n = F(F(theta) / tau), 200_000
            x = np.where(rng.random(n) < 0.2, rng.uniform(8 - 4e-4, 8 + 1e-4, n), rng.uniform(0.2, 8.2, n))
            t_next = (x * np.float64(tau)).astype(F)
            e_lo, _ = expf_range(t_next, tau)
            u = rng.uniform(-2.0, 24.0, n) * 2.0 ** -20
            delta = np.exp(rng.uniform(np.log(1e-6), 0.0, n))
            a, b = states_with_root_near(e_lo.astype(np.float64), u, delta, c)
            may = reference_may_accept(a, b, NO_T, t_next, c, tau, F(np.inf), conv=conv)
            claim = _claims(exe, conv, a, b, 0.0, e_lo, c, np.inf)
            assert not (claim & may).any()
            claims += int(claim.sum())
            planted += int((_claims(exe, conv, a, b, 0.0, e_lo * F(1 - 2.0 ** -14), c, np.inf) & may).sum())
            max_sim = F(rng.uniform(0.2, 8.0) * np.float64(tau))
            e_max = F(np.exp(np.float64(max_sim) / np.float64(tau)))
            a, b = states_with_root_near(np.full(n, np.float64(e_max)), u, delta, c)
            may = reference_may_accept(a, b, NO_T, F(np.inf), c, tau, max_sim, conv=conv)
            claim = _claims(exe, conv, a, b, 0.0, np.inf, c, e_max)
            assert not (claim & may).any()
            claims += int(claim.sum())
    assert claims > 100_000 and planted > 0, (claims, planted)


@pytest.mark.parametrize("conv", [False, True], ids=["fc", "conv"])
def test_claims_at_the_windows_start_are_never_accepted(exe, conv):
    """Smaller or larger root, or the vertex between two close roots, just before the event. Planted: a window that
    starts 2^-12 late."""
    rng = np.random.default_rng(22)
    claims = planted = 0
    for tau in TAUS:
        for theta in THETAS:
            for larger in (False, True):
                c, n = F(F(theta) / tau), 200_000
                t_ev = (rng.uniform(0.2, 8.05, n) * np.float64(tau)).astype(F)
                _, e_hi = expf_range(t_ev, tau)
                u = rng.uniform(-40.0, 4.0, n) * 2.0 ** -20
                delta = np.exp(rng.uniform(np.log(1e-12), 0.0, n))
                a, b = states_with_root_near(e_hi.astype(np.float64), u, delta, c, larger=larger)
                may = reference_may_accept(a, b, t_ev, F(np.inf), c, tau, F(np.inf), conv=conv)
                claim = _claims(exe, conv, a, b, e_hi, np.inf, c, np.inf)
                assert not (claim & may).any()
                claims += int(claim.sum())
                planted += int((_claims(exe, conv, a, b, e_hi * F(1 + 2.0 ** -12), np.inf, c, np.inf) & may).sum())
    assert claims > 100_000 and planted > 0, (claims, planted)


@pytest.mark.parametrize("conv", [False, True], ids=["fc", "conv"])
def test_claims_on_operands_of_every_class_are_never_accepted(exe, conv):
    """Random magnitudes, signs, zeros, subnormals, infinities and NaN, in windows over all times."""
    rng = np.random.default_rng(23)
    claims = 0
    for tau in TAUS:
        n = 400_000
        c = F(np.exp(rng.uniform(np.log(2.0 ** -30), np.log(2.0 ** 16))))
        a, b = _wild(rng, n), _wild(rng, n)
        near = rng.random(n) < 0.5
        a[near], b[near] = rng.normal(0, 30, int(near.sum())).astype(F), rng.normal(3, 30, int(near.sum())).astype(F)
        t_ev = (rng.uniform(-1.0, 9.0, n) * np.float64(tau)).astype(F)
        t_next = (t_ev + np.exp(rng.uniform(np.log(1e-6), 1.0, n)) * tau).astype(F)
        e_ev, e_nx = (np.exp(v.astype(np.float64) / tau).astype(F) for v in (t_ev, t_next))
        claim = _claims(exe, conv, a, b, e_ev, e_nx, c, np.inf)
        may = reference_may_accept(a, b, t_ev, t_next, c, tau, F(np.inf), conv=conv)
        nan = ~(np.isfinite(a) & np.isfinite(b))
        assert not (claim & (may | nan)).any()
        claims += int(claim.sum())
    assert claims > 100_000, claims


@pytest.mark.parametrize("conv", [0, 1], ids=["fc", "conv"])
def test_gated_solver_matches_the_reference_loop(tmp_path, conv):
    assert SOLVER.count("solve_candidate") == 1 and SOLVER.count("look") >= 3
    exe = _build(tmp_path, "solver", SOLVER)
    r = subprocess.run([exe, "4000000", str(conv)], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr
    words = r.stdout.split()
    assert words[0] == "0" and int(words[5].rstrip(";")) > 500_000 and int(words[9]) > 1_000_000, r.stdout
