"""The fp32 kernel at the edges of its tiles (64 keys), of its row blocks (8 and 16 rows) and of its fragments."""
import pytest
import torch

from inference_lib_b200 import _cabi
from inference_lib_b200 import workloads as wl
from oracle import hogwild_oracle as oracle
from tests.gpu_util import run_cabi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("E", [64, 128])
@pytest.mark.parametrize("W,G,S,lengths", [
    (1, 1, 1, [1]),                          # one row, one key
    (1, 8, 1, [64]),                         # exactly one tile, exactly the 8-row instantiation
    (3, 3, 1, [63, 65, 129, 7]),             # 9 rows; tiles one short, one over
    (2, 4, 2, [700, 90, 131]),               # 16 rows, causal pairs
    (2, 5, 7, [300, 200, 257]),              # 70 rows: blocks of 16, the last one with 6
])
@pytest.mark.parametrize("max_ctas", [0, 3])
def test_matches_the_oracle(E, W, G, S, lengths, max_ctas):
    orders = [[0]] if len(lengths) == 1 else None
    p = wl.make_problem("f32", W=W, Hq=2 * G, Hkv=2, E=E, S=S, lengths=lengths, theta=5e5, dtype=torch.float32, seed=3, orders=orders)
    ref, ref_rq = oracle.fused(p.queries, p.cos, p.sin, p.locations, p.keys, p.values, p.scale)
    r = run_cabi(p, want_rq=True, max_ctas=max_ctas)
    assert r.rc == 0 and r.status == 0
    assert torch.equal(r.rq.cpu(), ref_rq)
    # a sum of n products of unit normals, each rounded to 2^-24: the scores are off by up to 2 sqrt(E) 2^-24, a row's output
    # (weights that add up to one over values of at most 5) by five times that and the sums' own rounding
    err = float((r.out.cpu() - torch.nan_to_num(ref)).abs().max())
    assert err < 2e-5, err


def test_rows_past_the_true_length_are_not_touched():
    p = wl.make_problem("f32", W=2, Hq=8, Hkv=2, E=128, S=1, lengths=[300, 70, 71], theta=5e5, dtype=torch.float32, seed=4)
    ref, _ = oracle.fused(p.queries, p.cos, p.sin, p.locations, p.keys, p.values, p.scale)
    keys = [torch.cat([k, torch.full_like(k[:, :, :50], float("nan"))], 2).cuda() for k in p.keys]
    values = [torch.cat([v, torch.full_like(v[:, :, :50], float("nan"))], 2).cuda() for v in p.values]
    r = run_cabi(p, kernel=_cabi.KERNEL_FMA, keys=keys, values=values)
    assert r.rc == 0 and r.status == 0
    assert float((r.out.cpu() - ref).abs().max()) < 2e-5
