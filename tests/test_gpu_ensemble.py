"""Ensemble of independent cases (nse_ensemble_*): heterogeneous grids, masks
and precisions stepped together on several streams, the steps after the first
replayed from a captured CUDA graph.  Every case must end bit-identical to the
same case stepped on its own (same kernels in the same order per case), for
even and odd step counts."""
import numpy as np
import pytest

from tests.test_gpu_step import make_case
from vtkmakecompare_b200 import solver as S

pytestmark = pytest.mark.gpu

SHAPES = [((64, 48, 64), S.FP64), ((96, 48, 64), S.FP64), ((128, 40, 96), S.MIXED),
          ((64, 64, 64), S.MIXED), ((40, 33, 36), S.FP64)]
KEYS = ("u", "v", "w", "p", "T", "u_ta", "u_pre", "T_pre", "divu")


def make(n, prec, seed):
    g, f, c1, par = make_case(*n, seed=seed, sphere=True)
    cfg = S.Config(g["nx"], g["ny"], g["nz"], par["dt"], par["Re"], par["Sc"], par["eta"],
                   g["xl"], g["yl"], g["zl"], y0=-1.0, ystretch=2.0, body_force=par["force"],
                   heat_source=par["source"], t_bot=par["tbot"], t_top=par["ttop"],
                   t_solid=par["tsolid"], precision=prec)
    c = S.Context(cfg)
    for k in ("u", "v", "w", "T"):
        c.upload(k, f[k])
    c.upload("cellvalue", c1)
    c.project()
    c.start()
    return c


def test_ensemble_matches_cases_stepped_alone():
    ens_cases = [make(n, p, 10 + i) for i, (n, p) in enumerate(SHAPES)]
    solo = [make(n, p, 10 + i) for i, (n, p) in enumerate(SHAPES)]
    try:
        with S.Ensemble(ens_cases, nstreams=3) as ens:
            for n_steps in (7, 4, 1, 5):
                ens.step(n_steps)
                ens.sync()
                for c in solo:
                    c.step(n_steps)
                    c.sync()
                for i, (a, b) in enumerate(zip(ens_cases, solo)):
                    assert a.step_index == b.step_index
                    for k in KEYS:
                        assert np.array_equal(a.download(k), b.download(k)), (i, k, n_steps)
    finally:
        for c in ens_cases + solo:
            c.close()


# Calls of odd and even length: the first two make one graph.  Once all pairs have one,
# all but one step of an odd call, and the first where the temperature buffers are out
# of step, are replays, whatever the call before left.  Same bits as stepped alone.
def test_ensemble_calls_of_odd_length_replay_their_pairs():
    shapes = [((64, 48, 64), S.FP64), ((40, 33, 36), S.FP64)]
    ens_cases = [make(n, p, 20 + i) for i, (n, p) in enumerate(shapes)]
    solo = [make(n, p, 20 + i) for i, (n, p) in enumerate(shapes)]
    early, often, late = (7, 20), (7, 3, 5, 8) * 8, (7, 7, 5, 8, 9, 3, 4, 8, 3)
    init = [{key: c.download(key) for key in ("u", "v", "w", "T")} for c in solo]
    try:
        with S.Ensemble(ens_cases, nstreams=2) as ens:
            for k, n_steps in enumerate(early + often + late):
                if k % 12 == 11 and k < len(early + often):  # (300 steps on end blow up)
                    for c, f in zip(ens_cases + solo, init + init):
                        for key in f:
                            c.upload(key, f[key])
                        c.step_index = 1
                        c.start()
                g0, l0 = S.graph_count(), S.graph_count(True)
                ens.step(n_steps)
                ens.sync()
                made, pairs = S.graph_count() - g0, S.graph_count(True) - l0
                if k < len(early):  # a graph for the inner pairs in the first call, no more
                    assert made == int(k == 0) and pairs > 0, (k, n_steps, made, pairs)
                if k >= len(early + often):
                    assert made == 0 and 2 * pairs >= n_steps - 2, (k, n_steps, made, pairs)
                for c in solo:
                    c.step(n_steps)
                    c.sync()
                for i, (a, b) in enumerate(zip(ens_cases, solo)):
                    for key in KEYS if k % 9 == 0 or k >= len(early + often) else ("u",):
                        x = a.download(key)
                        assert np.isfinite(x).all(), (i, key, k)
                        assert np.array_equal(x, b.download(key)), (i, key, k)
    finally:
        for c in ens_cases + solo:
            c.close()


# A first call of one pair makes the graph of the pairs inside longer calls, so that the
# long call after it makes none.
@pytest.mark.parametrize("first", [2, 3])
def test_ensemble_long_call_after_a_short_one_makes_no_graph(first):
    cases = [make(n, p, 30 + i) for i, (n, p) in enumerate(SHAPES[-2:])]
    try:
        with S.Ensemble(cases, nstreams=2) as ens:
            ens.step(1)
            counts = []
            for n_steps in (first, 20):
                g0, l0 = S.graph_count(), S.graph_count(True)
                ens.step(n_steps)
                ens.sync()
                counts.append((S.graph_count() - g0, S.graph_count(True) - l0))
        assert counts[0][0] == 1 and counts[1][0] == 0 and counts[1][1] >= 8, counts
    finally:
        for c in cases:
            c.close()
