"""Who folds the partials of the tcgen05 kernel of two query tiles per block: the last CTA of a unit where no unit has more than three
and every CTA has a step, the merge step otherwise.  ``max_ctas`` CTAs cut the units of a small call into so many parts; the plan's list of what is left to the
merge step (its length is the workspace's first word) says which of the two it was."""
import ctypes as C

import pytest
import torch

from inference_lib_b200 import _cabi
from inference_lib_b200 import workloads as wl
from oracle import hogwild_oracle as oracle
from tests.gpu_util import check_against

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
TILE, FOLDED = 128, 3            # rows of a query tile and keys of a step; CTAs of a unit up to which the last of them folds


def _plan(blocks, Hkv, grid):
    """Where every CTA starts, and the first CTA and the number of CTAs of every unit; ``blocks``: (steps, one query tile)."""
    n = len(blocks)
    pos, parts = (C.c_int64 * (grid + 1))(), (C.c_int32 * (2 * n * Hkv))()
    assert _cabi.load().hogatt_dense_plan((C.c_int32 * n)(*[s for s, _ in blocks]), (C.c_uint8 * n)(*[int(x) for _, x in blocks]), n, Hkv,
                                          grid, pos, parts) == 0
    return list(pos), list(parts)[1::2]


def _blocks(tile_keys):
    """Steps of every block from the keys that every query tile sees of every fragment."""
    out = []
    for b in range(0, len(tile_keys), 2):
        pair = tile_keys[b:b + 2]
        per = TILE if len(pair) == 2 else 2 * TILE
        out.append((sum(-(-max(seen) // per) for seen in zip(*pair)), len(pair) == 1))
    return out


def _tiles(p):
    """The (worker, tokens) that a query tile holds."""
    G = p.Hq // p.Hkv
    rows = G * p.S
    if rows <= TILE:
        return [[(w, range(p.S)) for w in range(t, min(t + TILE // rows, p.W))] for t in range(0, p.W, TILE // rows)]
    if TILE % G == 0:
        return [[(w, range(s, min(s + TILE // G, p.S)))] for w in range(p.W) for s in range(0, p.S, TILE // G)]
    return [[(w, sorted({x % p.S for x in range(r, min(r + TILE, rows))}))] for w in range(p.W) for r in range(0, rows, TILE)]


def _left_to_the_merge_step(blocks, Hkv, grid):
    """How many units are, and how many CTAs work on each unit."""
    pos, parts = _plan(blocks, Hkv, grid)
    few = max(parts) <= FOLDED and all(p < pos[grid] for p in pos[:grid])
    return sum(n == 0 or (n > 1 and not few) for n in parts), parts


def _problem(W, G, S, Hkv, dtype, prompt):
    lengths = [prompt] + [S + 74 + 7 * w for w in range(W)]
    p = wl.make_problem("fold", W=W, Hq=G * Hkv, Hkv=Hkv, E=128, S=S, lengths=lengths, theta=5e5, dtype=dtype, seed=3)
    loc = p.locations.clone()
    loc[:, 0, 0] = -1                                       # a row that sees nothing
    if W > 1:
        loc[1:, W - 1] = -1                                 # a worker that sees the first fragment only
    return wl.Problem(**{**p.__dict__, "locations": loc})


def _bind(p, d, out, status, **kw):
    bp = _cabi.bind(out=out, queries=d.queries, locations=d.locations, keys=d.keys, values=d.values, scale=p.scale,
                    fragment_lengths=d.fragment_lengths, cos=d.cos, sin=d.sin, status=status, **kw)
    ws = _cabi.attach_workspace(bp, torch.device(DEV))
    ws.fill_(0xFF)                                          # (NaN where nothing has been left)
    first = bp.struct.workspace - ws.data_ptr()
    return bp, lambda: int(ws[first:first + 4].view(torch.int32).item())


@pytest.mark.parametrize("W,G,S,Hkv,dtype", [
    (2, 8, 16, 2, torch.bfloat16),                          # a worker is a tile
    (3, 8, 16, 1, torch.float16),                           # ... and the third one's block has one tile only
    (3, 8, 16, 2, torch.bfloat16),
    (1, 8, 48, 1, torch.bfloat16),                          # tiles of 16 tokens, three of them
    (2, 4, 64, 1, torch.float16),                           # tiles of 32 tokens, two per worker
    (1, 5, 128, 1, torch.bfloat16),                         # runs of 128 rows across heads, five of them
])
@pytest.mark.parametrize("max_ctas", [1, 2, 3, 4, 5, 7, 9])
def test_units_of_any_number_of_parts(W, G, S, Hkv, dtype, max_ctas):
    _check(_problem(W, G, S, Hkv, dtype, 3000), max_ctas)


@pytest.mark.parametrize("W,max_ctas,prompt", [
    (2, 9, 18500),                                          # one unit; the merge step's warps share its partials,
    (2, 31, 64000), (2, 32, 66000),                         # ... the last form without and the first with several of them in flight
    (2, 33, 68000), (3, 65, 67000),                         # two units, one of one query tile
])
def test_units_of_many_parts(W, max_ctas, prompt):
    _check(_problem(W, 8, 16, 1, torch.bfloat16, prompt), max_ctas)


def _check(p, max_ctas):
    dtype, Hkv = p.dtype, p.Hkv
    ref, _ = oracle.fused(p.queries, p.cos, p.sin, p.locations, p.keys, p.values, p.scale)
    d = p.to(DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    out = torch.full((p.W, p.Hq, p.S, p.Ev), float("nan"), dtype=dtype, device=DEV)
    bp, left = _bind(p, d, out, status, max_ctas=max_ctas)
    shape = _cabi.launch_shape(bp)
    assert shape["kernel"] == _cabi.KERNEL_DENSE and shape["kernels_per_call"] == 4        # plan, rotation, attention, merge
    lengths = torch.tensor([k.shape[-2] for k in p.keys], dtype=torch.int32)
    keys = [[max(max(0, min(int(p.locations[f, w, s]), int(lengths[f]) - 1) + 1) for w, tokens in tile for s in tokens) for f in range(p.F)]
            for tile in _tiles(p)]
    expected, _ = _left_to_the_merge_step(_blocks(keys), Hkv, max_ctas)
    results = []
    for _ in range(4):                                      # whichever CTA is the last one: the same bits
        out.fill_(float("nan"))
        assert _cabi.launch(bp, torch.cuda.current_stream().cuda_stream) == 0
        torch.cuda.synchronize()
        assert int(status.item()) == 0 and left() == expected
        results.append(out.clone())
    check_against(results[0], ref.numpy(), dtype, what=f"{max_ctas} CTAs")
    assert all(torch.equal(r, results[0]) for r in results[1:])


@pytest.mark.parametrize("max_ctas", [2, 3, 7])
def test_rows_that_are_stored_to_several_outputs(max_ctas):
    """A fused-gather call of rank 1 of two, its peer's flag already set: folded rows and merged ones go to both outputs."""
    full = _problem(2, 8, 16, 4, torch.bfloat16, 3000)
    p = full.shard(1, 2)
    ref, _ = oracle.fused(p.queries, p.cos, p.sin, p.locations, p.keys, p.values, p.scale)
    d = p.to(DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    own = torch.empty((p.W, p.Hq, p.S, p.Ev), dtype=p.dtype, device=DEV)
    bp, _ = _bind(p, d, own, status, max_ctas=max_ctas)
    outs = [torch.zeros((p.W, full.Hq, p.S, p.Ev), dtype=p.dtype, device=DEV) for _ in range(2)]
    flags = [torch.tensor([1, 0, 0], dtype=torch.int32, device=DEV) for _ in range(2)]
    peers = _cabi.Peers()
    peers.world, peers.rank = 2, 1
    for r in range(2):
        peers.out_full[r], peers.flags[r] = outs[r].data_ptr(), flags[r].data_ptr()
    assert _cabi.launch_gather(bp, peers, torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    for out in outs:
        check_against(out[:, p.Hq:], ref.numpy(), p.dtype, what=f"{max_ctas} CTAs")
        assert (out[:, :p.Hq] == 0).all()


@pytest.mark.parametrize("G,seqs,lens,least,most", [
    (4, [400, 1, 1], [700, 290, 33], 1, 3),                 # units of one to three parts, one tile in the last blocks
    (5, [300, 1, 1], [900, 290, 33], 1, 3),                 # 25 tokens per tile, three rows of it unused
    (4, [128], [500], 3, 3),                                # fewer steps than SMs
    (4, [256], [1000], 3, 5),                               # below and above what is folded
    (4, [64], [2000], 14, 14),
])
def test_packed_calls(G, seqs, lens, least, most):
    """Prompt chunks, two of them beside single tokens, whose units all SMs cut into few, some and many parts."""
    Hkv, bs, dtype, scale = 8, 16, torch.bfloat16, 128 ** -0.5
    grid = torch.cuda.get_device_properties(0).multi_processor_count
    per_tile, blocks = TILE // G, []
    for n, held in zip(seqs, lens):
        tiles = [[min(held, held - n + s + per_tile)] for s in range(0, n, per_tile)]
        blocks += _blocks(tiles)
    expected, parts = _left_to_the_merge_step(blocks, Hkv, grid)
    if grid == 148:
        assert (min(parts), max(parts)) == (least, most)
    gen = torch.Generator().manual_seed(lens[0])
    per = -(-max(lens) // bs)
    kc, vc = (torch.randn(len(seqs) * per, Hkv, bs, 128, generator=gen).to(dtype) for _ in range(2))
    table = torch.randperm(len(seqs) * per, generator=gen).to(torch.int32).reshape(len(seqs), per)
    table = torch.cat([table, torch.zeros(len(seqs), 2048 - per, dtype=torch.int32)], 1).contiguous()
    cu = torch.tensor([0] + [sum(seqs[:i + 1]) for i in range(len(seqs))], dtype=torch.int32)
    length = torch.tensor([lens], dtype=torch.int32)
    loc = torch.tensor([[n - s + t for n, s in zip(lens, seqs) for t in range(s)]], dtype=torch.int32)
    q = torch.randn(1, sum(seqs), Hkv * G, 128, generator=gen).to(dtype)
    ref = oracle.varlen_paged_sdpa(q, loc, length, kc, vc, table, cu, scale)
    d = [t.to(DEV) for t in (q, loc, length, kc, vc, table, cu)]
    out = torch.empty(sum(seqs), Hkv * G, 128, dtype=dtype, device=DEV)
    problem, keep = _cabi.bind_paged(out=out, queries=d[0], locations=d[1], fragment_lengths=d[2], key_cache=d[3], value_cache=d[4],
                                     block_table=d[5], scale=scale, cu_seqlens_q=d[6])
    ws, results = keep[0], []
    first = problem.workspace - ws.data_ptr()
    for _ in range(3):
        ws.fill_(0xFF)
        out.fill_(float("nan"))
        assert _cabi.launch_paged(problem, torch.cuda.current_stream().cuda_stream) == 0
        torch.cuda.synchronize()
        assert int(ws[first:first + 4].view(torch.int32).item()) == expected
        results.append(out.clone())
    check_against(results[0], ref.numpy(), dtype, what=f"{seqs} tokens of {lens} keys")
    assert all(torch.equal(r, results[0]) for r in results[1:])
