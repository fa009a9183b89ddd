"""The one-launch time step reuses its receive buffers on the strength of the exchanges between: this walks
the order that sends, landings and block barriers give between the eight CTAs of a cluster, with the
dealing of columns the kernel uses (csrc/step_deal.h, compiled here), and looks for a buffer, or a
barrier's next phase, that a peer may write before its last reader is done."""
import os
import subprocess

import pytest

from conftest import ROOT

RANKS = range(8)


@pytest.fixture(scope="module")
def deal(tmp_path_factory):
    d = tmp_path_factory.mktemp("deal")
    (d / "deal.cc").write_text("""#include <cstdio>
#include "step_deal.h"
int main() { for (int n = 16; n <= 1536; n += 16) { printf("%d", n); for (int r = 0; r <= 8; r++) printf(" %d", stepf::deal_from(n, r));
 printf(" %d", stepf::per_cta(n)); for (int f = 16; f <= 1536; f += 16) printf(" %d", stepf::exchanges_order_reuse(n, f)); puts(""); } }
""")
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "nncp-metal_b200", "csrc"), "-o", str(d / "deal"), str(d / "deal.cc")], check=True)
    rows = [list(map(int, line.split())) for line in subprocess.run([str(d / "deal")], capture_output=True, text=True, check=True).stdout.splitlines()]
    return {r[0]: (r[1:10], r[10], r[11:]) for r in rows}


def test_deal_covers_every_column_once(deal):
    for n, (at, most, _) in deal.items():
        assert at[0] == 0 and at[8] == n
        for r in RANKS:
            assert at[r] % 8 == 0 and 0 <= at[r + 1] - at[r] <= most
            assert n < 64 or at[r + 1] > at[r]


def unordered(deal, D, H, dk, F, nb):
    """Reuses without a path from the last read.  Nodes (event, layer, CTA); a CTA's events of a layer: Q, LQ the
    projection's sends and their landing, A attention and its sends, LO their landing, P1, LT1 the output
    projection, S5 the norm's block barrier, H, LH feed-forward up, P2, LT2 down, S9 the second norm's."""
    HD = H * dk
    cols = {"Q": deal[3 * HD][0], "P1": deal[D][0], "P2": deal[D][0], "H": deal[F][0]}
    barrier = not deal[HD][2][F // 16 - 1]
    has = lambda e, r: cols[e][r + 1] > cols[e][r]
    heads = [{p % H for p in range(r, nb * H, 8)} for r in RANKS]  # a CTA's (stream, head) pairs
    first, second = ("Q", "LQ", "A", "LO", "P1", "LT1", "S5"), ("H", "LH", "P2", "LT2", "S9")
    after = {}

    def edge(a, b):
        after.setdefault(a, []).append(b)

    for layer in (0, 1):
        for r in RANKS:
            n = lambda e: (e, layer, r)
            for a, b in (("LQ", "A"), ("LO", "P1"), ("LT1", "S5"), ("LH", "P2"), ("LT2", "S9")):
                edge(n(a), n(b))
            for e in first[:-2]:
                edge(n(e), n("S5"))
            for e in second:
                edge(n("S5"), n(e))
            for e in second[:-2]:
                edge(n(e), n("S9"))
            for z in RANKS if barrier else (r,):
                for e in second[:3]:
                    edge(n("S5"), (e, layer, z))
                for e in first:
                    edge(n("S9"), (e, layer + 1, z))
            for z in RANKS:
                if any((c % HD) // dk in heads[z] for c in range(cols["Q"][r], cols["Q"][r + 1], 4)):
                    edge(n("Q"), ("LQ", layer, z))
                if heads[r]:
                    edge(n("A"), ("LO", layer, z))
                for e, landing in (("P1", "LT1"), ("H", "LH"), ("P2", "LT2")):
                    if has(e, r):
                        edge(n(e), (landing, layer, z))
    paths = {}

    def reaches(a, b):
        if a not in paths:
            seen, todo = set(), [a]
            while todo:
                for y in after.get(todo.pop(), ()):
                    if y not in seen:
                        seen.add(y)
                        todo.append(y)
            paths[a] = seen
        return b in paths[a]

    bad = []
    for x in RANKS:      # reads, or waits for the phase
        for y in RANKS:  # writes
            want = []
            if has("P1", y):
                want += [("S5", "P2", 0), ("S9", "P1", 1), ("LT1", "P1", 1), ("LT2", "P2", 1)]
            if has("H", y):
                want += [("LH", "H", 1), ("S9", "H", 1)]
            if heads[y]:
                want += [("LO", "A", 1), ("S5", "A", 1)]
            if has("Q", y) and heads[x]:
                want += [("LQ", "Q", 1), ("A", "Q", 1)]
            bad += [(a, b, x, y) for a, b, later in want if (a, b) != ("S9", "H") or has("P2", x)
                    if (a, b) != ("S5", "A") or has("P1", x) if not reaches((a, 0, x), (b, later, y))]
    return bad


@pytest.mark.parametrize("H,dk", [(1, 16), (2, 8), (1, 32), (3, 16), (4, 16), (7, 16), (3, 32), (8, 32), (12, 4)])
def test_every_reuse_follows_its_last_read(deal, H, dk):
    for D in (16, 48, 64, 96, 112, 512):
        for F in (16, 48, 64, 96, 112, 208, 272):
            for nb in (1, 4):
                assert not unordered(deal, D, H, dk, F, nb), (D, F, nb)
