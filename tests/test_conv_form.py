"""The rule that gives a batch of the position-grouped conv backward to one of its two kernels (conv_events_pays,
bats_gb300/csrc/conv_form.cuh): it is the stated inequality in exact arithmetic, also where its products pass 64 bits; and one kernel
alone decides, since two that each decided could leave a batch to nobody."""
import ctypes
import os
import re
import shutil
import subprocess
from fractions import Fraction

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "bats_gb300", "csrc")


def load_rule(folder):
    """conv_events_pays as a host function of (spiking, events, samples, n_pos, taps, field)."""
    if shutil.which("g++") is None:
        pytest.skip("no host C++ compiler")
    src, lib = os.path.join(str(folder), "form.cpp"), os.path.join(str(folder), "form.so")
    with open(src, "w") as f:
        f.write('#include "conv_form.cuh"\nextern "C" int pays(unsigned long long a, unsigned long long b, int c, int d, int e, int f) '
                "{ return bats::conv_events_pays(a, b, c, d, e, f); }\n")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, "-o", lib, src], check=True)
    fn = ctypes.CDLL(lib).pays
    fn.argtypes = [ctypes.c_ulonglong, ctypes.c_ulonglong] + [ctypes.c_int] * 4
    return lambda *a: bool(fn(*a))


def test_rule_is_exact(tmp_path):
    rule = load_rule(tmp_path)
    rng = np.random.default_rng(3)
    seen = {True: 0, False: 0}
    for _ in range(20000):
        samples, n_pos, field = int(np.exp(rng.uniform(0, 11))), int(rng.integers(1, 256)), int(rng.integers(1, 50))
        taps = field * int(rng.integers(1, 1024 // field + 1))
        events = samples * int(np.exp(rng.uniform(0, 20)))
        work = Fraction(events * -(-taps // 32))
        chunks = Fraction(events, 32 * n_pos * samples) + Fraction(1, 2)
        line = Fraction(1, 3) * work / (chunks * field)
        spiking = max(0, int(line) + int(rng.integers(-2, 3))) if rng.random() < 0.7 else int(line * Fraction(rng.uniform(0, 2)))
        spiking = min(spiking, 2 ** 40)
        want = work >= 256 * samples and spiking * field * chunks <= Fraction(1, 3) * work
        assert rule(spiking, events, samples, n_pos, taps, field) == want
        seen[want] += 1
    assert min(seen.values()) > 3000, seen


def test_one_kernel_decides():
    text = open(os.path.join(CSRC, "conv_pool.cu")).read()
    kernels = re.split(r"\n(?=__global__|template <[^\n]*>\n__global__)", text)
    deciding = [k for k in kernels[1:] if re.search(r"[( ]conv_events_form(<\w+>)?\(", k.split("\n}\n")[0])]
    assert len(deciding) == 1, len(deciding)
