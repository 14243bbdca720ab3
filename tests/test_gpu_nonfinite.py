"""A NaN or an infinite score shows in the results it belongs to, whatever the position of the query or key, and
in no others."""
import numpy as np
import pytest
import torch

from flash_attention3_b200 import ops
from oracle import golden
from tests.helpers import dev, host

pytestmark = pytest.mark.gpu

# (heads, length): pairs of query tiles whose keys a cluster shares; pairs of the last and the first tile; neighbours
PROBLEMS = [(1, 640), (12, 449), (200, 1100)]
# tensor, row, value: rows of the first and of later tiles, keys with either form of the exponential at D=64
PLANTS = [("q", 3, np.nan), ("q", 200, np.nan), ("k", 3, np.nan), ("k", 14, np.nan), ("k", 159, np.nan),
          ("k", 14, np.inf), ("k", 64, np.inf)]


def planted(heads, s, d, name, row, value):
    q, k, v, do = golden.seeded_inputs(51, 1, heads, heads, s, d, "fp16")
    clean = {"q": q.copy(), "k": k.copy(), "v": v, "do": do}
    {"q": q, "k": k}[name][0, 0, row, 5] = value
    return clean, {"q": q, "k": k, "v": v, "do": do}


def bad_rows(x, causal_rows):
    """Rows of head 0 of a causal problem with a visible score that is NaN or +inf."""
    with np.errstate(invalid="ignore"):
        score = np.matmul(x["q"][0, 0], x["k"][0, 0].T)
    visible = np.tril(np.ones((causal_rows, causal_rows), bool))
    return ((np.isnan(score) | np.isposinf(score)) & visible).any(axis=1)


def check_forward(heads, s, d, plant, softcap):
    clean, x = planted(heads, s, d, *plant)
    bad = np.zeros((heads, s), bool)
    bad[0] = bad_rows(x, s)
    assert bad.any() and not bad.all()
    run = lambda t: ops.fa3_fwd(dev(t["q"], "fp16"), dev(t["k"], "fp16"), dev(t["v"], "fp16"), True, softcap=softcap, sync=True)
    out, lse = (host(t)[0] for t in run(x))
    assert np.isnan(out[bad]).all() and np.isnan(lse[bad]).all(), (np.isnan(out).sum(), np.isnan(lse).sum())
    assert np.isfinite(out[~bad]).all() and np.isfinite(lse[~bad]).all()
    if np.isnan(plant[2]):  # (an infinity also takes keys out of other rows)
        out0, lse0 = (host(t)[0] for t in run(clean))
        assert np.array_equal(out[~bad], out0[~bad]) and np.array_equal(lse[~bad], lse0[~bad])


@pytest.mark.parametrize("plant", PLANTS)
@pytest.mark.parametrize("heads,s", PROBLEMS)
@pytest.mark.parametrize("d", [64, 128])
def test_forward(d, heads, s, plant):
    check_forward(heads, s, d, plant, 0.0)


@pytest.mark.parametrize("plant", [p for p in PLANTS if np.isnan(p[2])])
@pytest.mark.parametrize("heads,s", PROBLEMS[:2])
@pytest.mark.parametrize("d", [64, 128])
def test_forward_softcap(d, heads, s, plant):
    check_forward(heads, s, d, plant, 20.0)


@pytest.mark.parametrize("name,row", [("q", 3), ("q", 200), ("k", 3), ("k", 159)])
@pytest.mark.parametrize("deterministic", [False, True])
@pytest.mark.parametrize("d", [64, 128])
def test_backward_softcap(d, deterministic, name, row):
    s = 300
    clean, x = planted(1, s, d, name, row, np.nan)
    t = {n: dev(a, "fp16") for n, a in x.items()}
    out, lse = ops.fa3_fwd(dev(clean["q"], "fp16"), dev(clean["k"], "fp16"), t["v"], True, softcap=20.0)
    dq, dk, dv = (host(g)[0, 0] for g in ops.fa3_bwd(t["do"], t["q"], t["k"], t["v"], out, lse, True, softcap=20.0,
                                                     deterministic=deterministic, sync=True))
    rows = np.arange(s)
    if name == "q":
        # the probabilities of one query row, over the keys it sees
        assert np.isnan(dq[row]).all() and np.isfinite(dq[rows != row]).all()
        assert np.isnan(dv[:row + 1]).all() and np.isfinite(dv[row + 1:]).all()
        assert np.isnan(dk[:row + 1]).all()  # (others: a zero times the NaN of Q)
    else:
        # the probabilities of one key, for the rows that see it
        assert np.isnan(dq[row:]).all()  # (others: a zero times the NaN of K)
        assert np.isnan(dv[row]).all() and np.isfinite(dv[rows != row]).all()
        assert np.isnan(dk[row]).all() and np.isfinite(dk[rows != row]).all()
