"""The tcgen05 kernel of two query tiles per block.  Few CTAs (``max_ctas``) make a small call long enough for it: every CTA gets
a step and a unit is cut into few parts."""
import pytest
import torch

from inference_lib_b200 import _cabi
from inference_lib_b200 import workloads as wl
from oracle import hogwild_oracle as oracle
from tests.gpu_util import check_against, run_cabi

pytestmark = pytest.mark.gpu


def _problem(W, G, S, lengths, dtype=torch.bfloat16, Hkv=2):
    orders = [[0]] if len(lengths) == 1 else None if len(lengths) == W + 1 else [list(range(len(lengths)))] * W
    return wl.make_problem("pairs", W=W, Hq=Hkv * G, Hkv=Hkv, E=128, S=S, lengths=lengths, theta=5e5, dtype=dtype, seed=6, orders=orders)


@pytest.mark.parametrize("W,G,S,lengths,dtype", [
    (1, 4, 320, [320], torch.bfloat16),                     # a causal prompt: tiles of 32 tokens x 4 heads, steps end with the tokens
    (1, 5, 128, [129], torch.float16),                      # G does not divide 128: runs of 128 rows across heads; five tiles, the last alone
    (3, 4, 32, [300, 40, 150, 257], torch.bfloat16),        # a tile per worker, three of them
    (9, 2, 8, [200, 9], torch.bfloat16),                    # eight workers in a tile, one in the second
    (2, 8, 16, [700, 128, 1], torch.float16),               # one block; fragments of whole and of single keys
    (2, 1, 256, [511, 300, 256], torch.bfloat16),           # a head per kv head
])
@pytest.mark.parametrize("max_ctas", [1, 2, 5])
def test_matches_the_oracle(W, G, S, lengths, dtype, max_ctas):
    p = _problem(W, G, S, lengths, dtype)
    loc = p.locations.clone()
    loc[:, 0, :2] = -1                                      # rows that see nothing at all
    if W > 1:
        loc[0, W - 1] = -1                                  # a worker that sees nothing of the first fragment
    p = wl.Problem(**{**p.__dict__, "locations": loc})
    ref, ref_rq = oracle.fused(p.queries, p.cos, p.sin, p.locations, p.keys, p.values, p.scale)
    for host_lengths in (None, "rows"):
        r = run_cabi(p, want_rq=True, max_ctas=max_ctas, host_lengths=host_lengths)
        assert r.rc == 0 and r.status == 0
        assert torch.equal(r.rq.cpu(), ref_rq)
        check_against(r.out, ref.numpy(), dtype, what=f"{W} {G} {S} {max_ctas} {host_lengths}")
    again = run_cabi(p, max_ctas=max_ctas, host_lengths="rows")
    assert torch.equal(again.out, r.out)


def test_many_parts_per_unit():
    """One unit cut into twenty parts: the merge step's warps share them."""
    p = _problem(2, 8, 16, [41000, 40, 90], Hkv=1)
    ref, _ = oracle.fused(p.queries, p.cos, p.sin, p.locations, p.keys, p.values, p.scale)
    r = run_cabi(p, max_ctas=20)
    assert r.rc == 0 and r.status == 0
    check_against(r.out, ref.numpy(), p.dtype)


def test_rows_past_the_true_length_never_reach_a_result():
    p = _problem(2, 4, 64, [300, 130, 257])
    ref, _ = oracle.fused(p.queries, p.cos, p.sin, p.locations, p.keys, p.values, p.scale)
    keys = [torch.cat([k, torch.full_like(k[:, :, :100], float("nan"))], 2).cuda() for k in p.keys]
    values = [torch.cat([v, torch.full_like(v[:, :, :100], float("inf"))], 2).cuda() for v in p.values]
    for max_ctas in (1, 3):
        r = run_cabi(p, keys=keys, values=values, max_ctas=max_ctas)
        assert r.rc == 0 and r.status == 0
        check_against(r.out, ref.numpy(), p.dtype)


def test_too_small_a_workspace_runs_on_the_other_kernel():
    p = _problem(1, 4, 320, [320])
    d = p.to("cuda:0")
    out = torch.empty((p.W, p.Hq, p.S, p.Ev), dtype=p.dtype, device="cuda:0")
    bp = _cabi.bind(out=out, queries=d.queries, locations=d.locations, keys=d.keys, values=d.values, scale=p.scale,
                    fragment_lengths=d.fragment_lengths, cos=d.cos, sin=d.sin, max_ctas=3)
    # ten 128-row units of at most five parts: rows of 128 values, a maximum and a sum, and the rotated queries behind them
    one_tile = 4096 + 20 * 5 * 128 * (128 + 2) * 4 + p.queries.numel() * 2
    ws = torch.empty(one_tile + 256, dtype=torch.uint8, device="cuda:0")
    bp.struct.workspace, bp.struct.workspace_bytes = ws.data_ptr() + (-ws.data_ptr()) % 256, one_tile
    assert _cabi.launch(bp, torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    ref, _ = oracle.fused(p.queries, p.cos, p.sin, p.locations, p.keys, p.values, p.scale)
    check_against(out, ref.numpy(), p.dtype)


@pytest.mark.parametrize("W,G,S,lengths,Hkv", [
    (1, 4, 160, [640, 360], 8),                             # five tiles: the last block holds one; shares of 1.9 steps
    (3, 4, 96, [400, 160, 160, 160], 4),
    (1, 8, 304, [700, 404], 2),
])
def test_every_partial_that_is_folded_has_been_written(W, G, S, lengths, Hkv):
    """On all SMs a share of a block of one tile can be shorter than its steps count for; the workspace is NaN beforehand."""
    p = _problem(W, G, S, lengths, Hkv=Hkv)
    ref, _ = oracle.fused(p.queries, p.cos, p.sin, p.locations, p.keys, p.values, p.scale)
    r = run_cabi(p)
    assert r.rc == 0 and r.status == 0
    check_against(r.out, ref.numpy(), p.dtype)


@pytest.mark.parametrize("W,G,S,lengths", [(2, 4, 64, [300, 130, 257]), (1, 4, 160, [290])])
@pytest.mark.parametrize("with_lengths", [False, True])
def test_rows_that_nobody_sees_never_reach_a_result(W, G, S, lengths, with_lengths):
    """Fragments that hold more rows than any query sees (no lengths given, or lengths that count those rows)."""
    p = _problem(W, G, S, lengths)
    loc = torch.minimum(p.locations, torch.tensor(lengths, dtype=torch.int32)[:, None, None] - 1)      # (else a row sees all there is)
    p = wl.Problem(**{**p.__dict__, "locations": loc})
    ref, _ = oracle.fused(p.queries, p.cos, p.sin, p.locations, p.keys, p.values, p.scale)
    more = [torch.cat([t, torch.full_like(t[:, :, :100], float("nan"))], 2) for t in p.keys + p.values]
    d = p.to("cuda:0")
    keys, values = [t.cuda() for t in more[:p.F]], [t.cuda() for t in more[p.F:]]
    rows = torch.tensor([k.shape[2] for k in keys], dtype=torch.int32, device="cuda:0") if with_lengths else None
    for max_ctas in (1, 3, 0):
        out = torch.full((p.W, p.Hq, p.S, p.Ev), float("nan"), dtype=p.dtype, device="cuda:0")
        bp = _cabi.bind(out=out, queries=d.queries, locations=d.locations, keys=keys, values=values, scale=p.scale, fragment_lengths=rows,
                        cos=d.cos, sin=d.sin, max_ctas=max_ctas)
        _cabi.attach_workspace(bp, torch.device("cuda:0"))
        assert _cabi.launch(bp, torch.cuda.current_stream().cuda_stream) == 0
        torch.cuda.synchronize()
        check_against(out, ref.numpy(), p.dtype, what=f"{max_ctas} CTAs")


@pytest.mark.parametrize("W,G,S,lengths", [(1, 4, 160, [290]), (4, 4, 8, [260, 33, 20, 70, 129])])
@pytest.mark.parametrize("scale", [0.0, -0.05, 1e-40])
def test_scales_that_are_not_positive(W, G, S, lengths, scale):
    """AUTO keeps such calls off both tcgen05 kernels.  (The oracle masks before it scales: negated queries, or none.)"""
    p = _problem(W, G, S, lengths)
    q = -p.queries if scale < -0.01 else torch.zeros_like(p.queries)
    ref, _ = oracle.fused(q, p.cos, p.sin, p.locations, p.keys, p.values, max(0.01, -scale))
    for max_ctas in (0, 2):
        r = run_cabi(wl.Problem(**{**p.__dict__, "scale": scale}), max_ctas=max_ctas)
        assert r.rc == 0 and r.status == 0
        check_against(r.out, ref.numpy(), p.dtype)


def test_a_workspace_asked_for_before_the_scale_is_known_is_enough():
    p = _cabi.shape_problem(F=1, W=1, Hq=32, Hkv=8, E=128, Ev=128, S=512, dtype=_cabi.BF16)
    q = _cabi.shape_problem(F=1, W=1, Hq=32, Hkv=8, E=128, Ev=128, S=512, dtype=_cabi.BF16, scale=0.0)
    lib = _cabi.load()
    assert lib.hogatt_workspace_bytes(q) >= lib.hogatt_workspace_bytes(p) > 0
