"""The dataflow factorization's own tile layout (df_layout, compiled here) under
the model of its programs in test_factor_schedule: every tile is owned once, by
a CTA whose program takes it, and every schedule ends; on the whole chip and on
parts of it."""
import os
import random
import subprocess

import pytest

from test_factor_schedule import Run, helper_cta, row_cta, worker

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "hs_sfm_gb300", "csrc")


@pytest.fixture(scope="module")
def layout(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("layout") / "factor_layout")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-I", CSRC, os.path.join(HERE, "cpp", "factor_layout.cpp"),
                    "-o", exe], check=True)

    def run(nt, mixed, sms):
        out = subprocess.run([exe], input=f"{nt} {int(mixed)} {sms}", capture_output=True, text=True, check=True)
        lines = out.stdout.split("\n")
        g, rows, helpers, most = map(int, lines[0].split())
        own = [[tuple(map(int, t.split(","))) for t in line.split()] for line in lines[1:1 + g]]
        return g, rows, helpers, most, own

    return run


@pytest.mark.parametrize("mixed", [True, False])
@pytest.mark.parametrize("sms", [152, 132, 76, 38, 7])
def test_layout_and_schedule(layout, mixed, sms):
    for nt in (2, 3, 4, 5, 7, 8, 9, 15, 19, 20, 37, 38, 39, 50, 75, 76, 77, 90):
        g, rows, helpers, most, own = layout(nt, mixed, sms)
        assert g == min(sms, nt * (nt + 1) // 2) and len(own) == g and most == max(map(len, own))
        assert rows in (0, nt) and helpers in (0, nt) and rows >= helpers and rows + helpers <= g
        assert sorted(t for o in own for t in o) == [(i, j) for i in range(nt) for j in range(i + 1)]
        r, ctas = Run(nt), []
        for c, tiles in enumerate(own):
            assert tiles == sorted(tiles, key=lambda t: (t[1], t[0]))
            if c < rows:      # the row's last tiles, a fixed number of them
                kept = 3 if mixed else 2
                assert tiles == [(c, j) for j in range(max(0, c + 1 - kept), c + 1)]
                ctas.append(row_cta(r, c, tiles))
            elif c < rows + helpers:
                i = c - rows
                assert tiles == [(i, j) for j in range(max(0, i - 5), max(0, i - 2))]
                if tiles:
                    ctas.append(helper_cta(r, i, tiles))
            elif rows:        # two independent halves, no diagonal tiles
                assert all(i != j for i, j in tiles)
                ctas += [worker(r, tiles[0::2]), worker(r, tiles[1::2])]
            else:
                ctas.append(worker(r, tiles))
        rng = random.Random(nt)
        # a round in which some CTA can go on applies or publishes one tile at least
        for _ in range(nt * (nt + 1) * (nt + 2) // 6 + 3 * nt * (nt + 1)):
            rng.shuffle(ctas)
            live = []
            for c in ctas:
                try:
                    next(c)
                    live.append(c)
                except StopIteration:
                    pass
            ctas = live
            if not ctas:
                break
        assert not ctas, (nt, sms)
        assert r.flags == {(i, j) for i in range(nt) for j in range(i + 1)} and len(r.y) == nt
