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


@pytest.mark.parametrize("E,rotary_dim", [(64, 64), (64, 32), (64, 12), (128, 128), (128, 40), (128, 2)])
@pytest.mark.parametrize("G,shift", [(4, 0), (4, 1), (9, 1), (9, 2)])
def test_rotation_of_the_queries(E, rotary_dim, G, shift):
    """Part of a head, halves that are no whole 16-byte pieces, tables off the 16-byte boundary; 8 and 16 rows; the call of queries
    that have been rotated before gives the same bits."""
    p = wl.make_problem("f32", W=1, Hq=2 * G, Hkv=2, E=E, S=1, lengths=[70, 65], theta=1e4, dtype=torch.float32, seed=5, rotary_dim=rotary_dim)
    ref, ref_rq = oracle.fused(p.queries, p.cos, p.sin, p.locations, p.keys, p.values, p.scale)
    dev, d = torch.device("cuda:0"), p.to("cuda:0")
    tables = []
    for t in (d.cos, d.sin):
        room = torch.empty(t.numel() + 4, device=dev)
        room[shift:shift + t.numel()] = t.flatten()
        tables.append(room[shift:shift + t.numel()].view(t.shape))
    out, again = (torch.full((p.W, p.Hq, p.S, E), float("nan"), device=dev) for _ in range(2))
    rq = torch.full(ref_rq.shape, float("nan"), device=dev)
    for fused in (True, False):
        bp = _cabi.bind(out=out if fused else again, queries=d.queries if fused else rq, locations=d.locations, keys=d.keys, values=d.values,
                        scale=p.scale, fragment_lengths=d.fragment_lengths, cos=tables[0] if fused else None, sin=tables[1] if fused else None,
                        rq=rq if fused else None)
        _cabi.attach_workspace(bp, dev)
        assert _cabi.launch(bp, torch.cuda.current_stream().cuda_stream) == 0
        torch.cuda.synchronize()
    assert torch.equal(rq.cpu(), ref_rq) and torch.equal(out, again)
    assert float((out.cpu() - ref).abs().max()) < 2e-5
