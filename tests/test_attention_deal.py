"""Which kernel and how many CTAs an attention launch takes (csrc/attention_deal.h, compiled here), against what was
measured on the device for both sides."""
import os
import subprocess

import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def deal(tmp_path_factory):
    d = tmp_path_factory.mktemp("attention_deal")
    (d / "deal.cc").write_text("""#include <cstdio>
#include <cstring>
#include "attention_deal.h"
int main() { char what[16]; long a, b, c, d, e; while (scanf("%15s %ld %ld %ld %ld %ld", what, &a, &b, &c, &d, &e) == 6)
 if (!strcmp(what, "adjoint")) printf("%d\\n", (int)attn::adjoint_by_128((int)a, b, (int)c, (int)d, (int)e)); }
""")
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "nncp-metal_b200", "csrc"), "-o", str(d / "deal"), str(d / "deal.cc")], check=True)

    def ask(what, rows):
        text = "".join("%s %d %d %d %d %d\n" % (what, *(tuple(r) + (0,) * 5)[:5]) for r in rows)
        return list(map(int, subprocess.run([str(d / "deal")], input=text, capture_output=True, text=True, check=True).stdout.split()))

    return ask


# head size, queries, first and last 64-key block: per number of pairs the warp-level kernel's time over the other's
ADJOINT = [
    (64, 16, 0, 0, {100: 1.17, 148: 1.16, 152: 0.71, 256: 0.74, 592: 0.78, 1024: 0.85}),
    (64, 32, 0, 0, {100: 1.10, 148: 1.09, 152: 0.76, 256: 0.77, 592: 0.80, 1024: 0.85}),
    (64, 64, 0, 0, {100: 1.18, 148: 1.20, 152: 0.84, 256: 0.88, 592: 0.90, 1024: 0.99}),
    (64, 16, 0, 2, {100: 1.36, 152: 0.92, 200: 0.94, 296: 0.96, 400: 1.14, 592: 1.00, 1024: 1.13}),
    (64, 32, 0, 1, {100: 1.48, 152: 1.08, 256: 1.08, 592: 1.11, 1024: 1.06}),
    (64, 64, 0, 1, {100: 1.53, 152: 1.22, 256: 1.19, 592: 1.21, 1024: 1.17}),
    (64, 64, 0, 2, {100: 1.45, 152: 1.21, 256: 1.17, 592: 1.24, 1024: 1.25}),
    (64, 16, 0, 3, {100: 1.64, 152: 1.15, 256: 1.17, 592: 1.24, 1024: 1.31}),
    (64, 64, 0, 4, {100: 1.58, 152: 1.30, 256: 1.29, 592: 1.27, 1024: 1.32}),
    (128, 16, 0, 0, {100: 1.14, 152: 1.14, 256: 1.18, 592: 1.24, 1024: 1.27}),
    (128, 64, 0, 1, {100: 1.75, 152: 1.76, 256: 1.78, 592: 1.64, 1024: 1.60})]


def test_adjoint_takes_the_kernel_that_measured_faster(deal):
    for dk, T, lo, hi, times in ADJOINT:
        for pairs, got in zip(times, deal("adjoint", [(dk, p, T, lo, hi) for p in times])):
            assert got == (times[pairs] >= 1.0), (dk, T, lo, hi, pairs)
    # a window of two 64-key blocks that lie in two 128-key blocks counts as two of one
    assert deal("adjoint", [(64, 256, 64, 1, 2), (64, 256, 64, 2, 3), (64, 148, 64, 1, 2)]) == [0, 1, 1]
