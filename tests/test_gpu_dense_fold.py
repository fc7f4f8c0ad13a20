"""Who folds the partials of the tcgen05 kernel of two query tiles per block: the last CTA of a unit up to three of them, the merge
step above that.  One kv head and ``max_ctas`` CTAs cut one unit, or a unit of two tiles and one of one, into so many parts."""
import pytest
import torch

from inference_lib_b200 import workloads as wl
from oracle import hogwild_oracle as oracle
from tests.gpu_util import check_against, run_cabi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,Hkv,dtype", [(2, 1, torch.bfloat16), (3, 1, torch.float16), (3, 2, torch.bfloat16), (1, 1, torch.bfloat16)])
@pytest.mark.parametrize("max_ctas", [1, 2, 3, 4, 5, 9])
def test_units_of_any_number_of_parts(W, Hkv, dtype, max_ctas):
    # a worker is a tile of 128 rows (8 heads x 16 tokens); one worker alone: 8 heads x 40 tokens, three tiles
    S = 16 if W > 1 else 40
    lengths = [3000] + [90 + 7 * w for w in range(W)]
    p = wl.make_problem("fold", W=W, Hq=8 * Hkv, Hkv=Hkv, E=128, S=S, lengths=lengths, theta=5e5, dtype=dtype, seed=3)
    loc = p.locations.clone()
    loc[:, 0, 0] = -1                                       # a row that sees nothing
    loc[1:, W - 1] = -1                                     # a worker that sees the first fragment only
    p = wl.Problem(**{**p.__dict__, "locations": loc})
    ref, _ = oracle.fused(p.queries, p.cos, p.sin, p.locations, p.keys, p.values, p.scale)
    r = run_cabi(p, max_ctas=max_ctas)
    assert r.rc == 0 and r.status == 0
    check_against(r.out, ref.numpy(), dtype, what=f"{W} workers, {max_ctas} CTAs")
    for _ in range(3):                                      # whichever CTA is the last one: the same bits
        assert torch.equal(run_cabi(p, max_ctas=max_ctas).out, r.out)
