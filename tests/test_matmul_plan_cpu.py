"""The plans of the tcgen05 matmuls and the division of their work between CTAs: the library's own header, compiled for the host.  Every
tile holds tokens and rows, the tiles cover the result once, the CTAs' ranges cover the tiles' slabs once, and the CTAs that share a cut
tile agree on its ticket and on the places of their shares."""
from __future__ import annotations

import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

from tests.util import KIND_Q4_K, KIND_Q6_K, KIND_Q8_0

SMS = (148, 132, 7, 1)


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = tmp_path_factory.mktemp("plan") / "matmul_plan.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-Wall", "-shared", "-fPIC", str(Path(__file__).with_name("matmul_plan.cpp")), "-o", str(out)], check=True)
    return C.CDLL(str(out))


def ints(values):
    return (C.c_int * len(values))(*(int(v) for v in values))


@pytest.mark.parametrize("kind", [KIND_Q4_K, KIND_Q6_K, KIND_Q8_0])
def test_plans(lib, kind):
    """Token counts around the tile widths, and large ones whose tiles, rounded up to 16 columns, are fewer than the plan asked for."""
    rng = np.random.default_rng(kind)
    tokens = [1, 9, 16, 17, 63, 64, 65, 129, 255, 256, 257, 300, 511, 513, 1000, 2047, 2689, 3073, 3100, 3120, 3121, 3585, 4161, 4200, 8000]
    tokens += [int(t) for t in np.exp(rng.uniform(0, np.log(9000), 150))]
    for T in tokens:
        shapes = [(256, [1]), (1536, [4700]), (1024, [9400]), (2048, [2400, 2300]), (14336, [4096]), (4096, [14336, 14336])]
        shapes += [(int(rng.integers(1, 9000)), [int(f) for f in np.exp(rng.uniform(0, np.log(30000), rng.integers(1, 5)))]) for _ in range(4)]
        for K, F in shapes:
            for sms in SMS if T < 1000 else SMS[:1]:
                rc = lib.check_plan(0, kind, T, K, ints(F), len(F), sms)
                assert rc == 0, (rc, kind, T, K, F, sms)


@pytest.mark.parametrize("kind", [KIND_Q4_K, KIND_Q6_K])
def test_integer_plans(lib, kind):
    rng = np.random.default_rng(kind)
    for T in (1, 3, 5, 8, 9, 16, 17, 33, 64):
        for _ in range(60):
            K, F = int(rng.integers(1, 16000)), [int(f) for f in np.exp(rng.uniform(0, np.log(30000), rng.integers(1, 5)))]
            if rng.random() < 0.3:  # about as many tiles as clusters of four or eight find SMs
                F = [128 * int(rng.choice([14, 15, 16, 18, 32, 33, 34, 37, 38]))]
            for sms in SMS:
                rc = lib.check_plan(1, kind, T, K, ints(F), len(F), sms)
                assert rc == 0, (rc, kind, T, K, F, sms)


@pytest.mark.parametrize("kind,integer", [(KIND_Q4_K, 0), (KIND_Q6_K, 0), (KIND_Q8_0, 0), (KIND_Q4_K, 1), (KIND_Q6_K, 1)])
def test_whole_tiles(lib, kind, integer):
    """Plans that deal whole tiles: more tiles than CTAs, as many, fewer."""
    rng = np.random.default_rng(kind)
    several = 0
    for T in (1, 9, 16) if integer else (1, 17, 39, 64, 65, 257, 512, 2048):
        shapes = [(256, [1]), (2304, [17920, 17920]), (1536, [25600, 25600]), (4096, [14336, 14336]), (512, [128 * 148]), (512, [128 * 149])]
        shapes += [(int(rng.integers(1, 9000)), [int(f) for f in np.exp(rng.uniform(0, np.log(60000), rng.integers(1, 5)))]) for _ in range(40)]
        for K, F in shapes:
            for sms in SMS:
                rc = lib.check_whole(integer, kind, T, K, ints(F), len(F), sms)
                assert rc <= 0, (rc, kind, T, K, F, sms)
                several += rc == 0 and sum((f + 127) // 128 for f in F) > sms
    assert several > 20


@pytest.mark.parametrize("bn", [16, 64, 128, 256])
def test_groups(lib, bn):
    """Groups of any size, empty ones and all empty ones among them."""
    rng = np.random.default_rng(bn)
    for _ in range(300):
        groups = int(rng.integers(1, 20))
        counts = [int(c) for c in rng.integers(0, rng.choice([2, 20, 70, 300, 900]), groups)]
        F = [int(f) for f in rng.integers(1, 2000, rng.integers(1, 3))]
        rc = lib.check_groups(int(rng.integers(1, 20)), ints(counts), groups, ints(F), len(F), bn, int(rng.choice(SMS)))
        assert rc == 0, (rc, counts, F)
