"""The stage-unit spans of the mma.sync matmul (csrc/gemm_i8.cu): CTA c of C takes the units [i8_span_begin(c), i8_span_begin(c + 1)), and
the CTAs that share a row group are found with i8_owner.  The library's own functions (csrc/gemm_plan.h), compiled for the host, against a
brute-force search over many (units, CTAs)."""
from __future__ import annotations

from tests.test_matmul_plan_cpu import lib  # noqa: F401


def test_owner_matches_a_search_over_the_spans(lib):  # noqa: F811
    for SU in list(range(1, 70)) + [148, 149, 512, 1000, 3584, 28672]:
        for C in (1, 2, 3, 7, 64, 132, 148):
            if C > SU:
                continue
            spans = [(lib.i8_begin(SU, c, C), lib.i8_begin(SU, c + 1, C)) for c in range(C)]
            assert spans[0][0] == 0 and spans[-1][1] == SU and all(b > a for a, b in spans)
            assert all(a == b for (_, a), (b, _) in zip(spans, spans[1:]))
            step = max(1, SU // 500)
            for x in list(range(0, SU, step)) + [SU - 1]:
                want = next(c for c, (a, b) in enumerate(spans) if a <= x < b)
                assert lib.i8_holder(SU, x, C) == want, (SU, C, x)
