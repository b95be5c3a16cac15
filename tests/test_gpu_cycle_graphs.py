"""Cycle graphs with different numbers of leading unconditional steps: which one runs changes no result.
Enough solves for a solver to add graphs, against the straight graph, bit by bit, with values that
change in between."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _system(n):
    rng = np.random.default_rng(n)
    i = np.arange(n)
    cols = i[:, None] + np.array([-1, 0, 1])
    ok = (cols >= 0) & (cols < n)
    rp = np.concatenate([[0], np.cumsum(ok.sum(1))]).astype(np.int32)
    vals = rng.uniform(-1.0, 1.0, cols.shape)
    vals[:, 1] = rng.uniform(2.2, 3.0, n)
    return rp, cols[ok].astype(np.int32), vals[ok], rng.standard_normal(n)


@pytest.mark.parametrize("restart", [3, 10, 50])
@pytest.mark.parametrize("precond", [1, 2])
@pytest.mark.parametrize("precision", [0, 1])
def test_added_graphs_change_nothing(gpu_ctx, monkeypatch, restart, precond, precision):
    from vfvchem_vfvm3d_b200 import GmresOptions, Pattern
    rp, ci, va, b = _system(5000)
    # few steps, more, few again: the wanted lead moves and comes back
    factors = [1.0] * 9 + [0.4] * 9 + [1.0] * 4 + [1.7] * 2

    def passes():
        p = Pattern.from_csr(gpu_ctx, rp, ci)
        off = np.repeat(np.arange(5000), np.diff(rp)) != ci
        out = []
        for f in factors:
            p.set_values(np.where(off, f * va, va))
            x, info = p.solve(b, None, GmresOptions(tol=1e-10, restart=restart, max_outer=300, precond=precond, precision=precision,
                                                    inner_rtol=1e-4, engine=1))
            assert info.status == 0
            out.append((x, info.iters, info.relres))
        return out

    many = passes()
    monkeypatch.setenv("VFV_STRAIGHT_GRAPH", "1")
    straight = passes()
    for (x, it, rel), (xs, its, rels) in zip(many, straight):
        assert it == its and rel == rels and np.array_equal(x, xs)
    # the same values again: the same result, whatever graph the solver has come to
    assert np.array_equal(many[0][0], many[8][0]) and np.array_equal(many[0][0], many[21][0])
