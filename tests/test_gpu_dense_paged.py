"""Packed queries over a paged cache on the tcgen05 kernel: AUTO's choice once the prompt chunks of a batch fill a query tile."""
import os
import subprocess
import sys

import numpy as np
import pytest
import torch

from inference_lib_b200 import _cabi
from oracle import hogwild_oracle as oracle
from tests.gpu_util import check_against

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dtype,G,bs,seqs,lens", [
    (torch.bfloat16, 4, 16, [65, 1, 0, 40, 64], [200, 129, 77, 40, 64]),     # 64 tokens are a block of two tiles
    (torch.bfloat16, 5, 8, [81, 1, 26], [300, 513, 127]),                    # 25 tokens per tile, 3 rows of it unused
    (torch.float16, 1, 32, [513, 3], [513, 400]),                            # a tile is 128 tokens
    (torch.bfloat16, 7, 256, [75, 2], [700, 259]),                           # cache blocks of two key tiles
    (torch.float16, 128, 64, [5, 1], [90, 256]),                             # a tile is one token
])
@pytest.mark.parametrize("F", [1, 2])
def test_prompt_chunks_match_the_oracle(dtype, G, bs, seqs, lens, F):
    rng = np.random.default_rng(G * 100 + bs)
    W, Hkv, E = len(seqs), 2, 128
    cu = torch.tensor([0] + list(np.cumsum(seqs)), dtype=torch.int32)
    total = int(cu[-1])
    gen = torch.Generator().manual_seed(G)
    per = max(lens) // bs + 2
    kc, vc = (torch.randn(W * per, Hkv, bs, E, generator=gen).to(dtype) for _ in range(2))
    table = torch.from_numpy(rng.permutation(W * per).astype(np.int32)).reshape(W, per)
    # (room in the table for the keys that make AUTO take the kernel)
    columns = max(per, int(4.5e6 / ((total - W) * Hkv * G * bs)) + 1)
    table = torch.cat([table, torch.zeros(W, columns - per, dtype=torch.int32)], 1).contiguous()
    length = torch.tensor([[max(1, n - 13 * f) for n in lens] for f in range(F)], dtype=torch.int32)
    loc = torch.tensor([[int(length[f, w]) - s + t for w, s in enumerate(seqs) for t in range(s)] for f in range(F)], dtype=torch.int32)
    loc[0, 0] = -1 if F == 2 else loc[0, 0]                                  # a row that sees nothing of one fragment
    rq = torch.randn(F, total, Hkv * G, E, generator=gen).to(dtype)
    ref = oracle.varlen_paged_sdpa(rq, loc, length, kc, vc, table, cu, E ** -0.5)
    # rows of the last cache block past a sequence's end may hold anything
    for w in range(W):
        n = int(length[:, w].max())
        for x in range(n, per * bs):
            vc[table[w, x // bs], :, x % bs] = float("nan")
            kc[table[w, x // bs], :, x % bs] = float("inf")
    dev = [t.to(DEV) for t in (rq, loc, length, kc, vc, table, cu)]
    outs = []
    for kernel in (_cabi.KERNEL_AUTO, _cabi.KERNEL_MMA):                     # the general path over the same inputs
        out = torch.full((total, Hkv * G, E), float("nan"), dtype=dtype, device=DEV)
        rc, keep = _cabi.paged_sdpa(out=out, queries=dev[0], locations=dev[1], fragment_lengths=dev[2], key_cache=dev[3], value_cache=dev[4],
                                    block_table=dev[5], scale=E ** -0.5, cu_seqlens_q=dev[6], kernel=kernel,
                                    stream=torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        assert rc == 0
        check_against(out, ref.numpy(), dtype, what=f"kernel {kernel}")
        outs.append(out.float())
    assert float((outs[0] - outs[1]).abs().max()) <= 2e-2


def test_which_calls_take_it():
    """The workspace tells the routes apart: enough chunk tokens beyond one per sequence for the room in the block table, the
    cache's extent known, blocks of whole swizzle groups."""
    p = _cabi.PagedProblem()
    p.F, p.W, p.Hq, p.Hkv, p.E, p.Ev = 1, 4, 16, 4, 128, 128
    p.dtype, p.cu_seqlens_q = _cabi.BF16, 1
    lib = _cabi.load()

    def need(**kw):
        for k, v in dict(dict(total_q_tokens=300, num_blocks=256, block_size=16, max_blocks_per_seq=64, kernel=_cabi.KERNEL_AUTO), **kw).items():
            setattr(p, k, v)
        return lib.hogatt_paged_workspace_bytes(p)

    def general(**kw):
        return need(**dict(kw, kernel=_cabi.KERNEL_MMA))

    assert need() != general()
    for kw in (dict(num_blocks=0), dict(block_size=12, max_blocks_per_seq=90), dict(block_size=4, max_blocks_per_seq=300),
               dict(total_q_tokens=270), dict(max_blocks_per_seq=58), dict(total_q_tokens=60, max_blocks_per_seq=4096)):
        assert need(**kw) == general(**kw)
    assert need(total_q_tokens=70, max_blocks_per_seq=4096) != general(total_q_tokens=70, max_blocks_per_seq=4096)


def _packed(dtype, Hkv, G, bs, seqs, lens, room, seed=3):
    """A packed batch on the device, its table as wide as `room` keys, and what the oracle says of it."""
    W, E = len(seqs), 128
    gen = torch.Generator().manual_seed(seed)
    cu = torch.tensor([0] + list(np.cumsum(seqs)), dtype=torch.int32)
    per = -(-max(lens) // bs)
    kc, vc = (torch.randn(W * per, Hkv, bs, E, generator=gen).to(dtype) for _ in range(2))
    table = torch.randperm(W * per, generator=gen).to(torch.int32).reshape(W, per)
    table = torch.cat([table, torch.zeros(W, max(0, -(-room // bs) - per), dtype=torch.int32)], 1).contiguous()
    length = torch.tensor([lens], dtype=torch.int32)
    loc = torch.tensor([[n - s + t for n, s in zip(lens, seqs) for t in range(s)]], dtype=torch.int32)
    rq = torch.randn(1, int(cu[-1]), Hkv * G, E, generator=gen).to(dtype)
    names = ("queries", "locations", "fragment_lengths", "key_cache", "value_cache", "block_table", "cu_seqlens_q")
    return dict(zip(names, (rq, loc, length, kc, vc, table, cu)))


def _run(p, scale, kernel=_cabi.KERNEL_AUTO):
    """One call with the workspace and the output filled with NaN."""
    d = {k: v.to(DEV) for k, v in p.items()}
    out = torch.full(p["queries"].shape[1:], float("nan"), dtype=p["queries"].dtype, device=DEV)
    problem, keep = _cabi.bind_paged(out=out, scale=scale, kernel=kernel, **d)
    keep[0].fill_(0xFF)
    assert _cabi.launch_paged(problem, torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    return out


def _oracle(p, scale):
    return oracle.varlen_paged_sdpa(*(p[k] for k in ("queries", "locations", "fragment_lengths", "key_cache", "value_cache", "block_table",
                                                     "cu_seqlens_q")), scale)


@pytest.mark.parametrize("Hkv,G,seqs,lens", [
    (2, 4, [367, 1, 1], [1675, 1666, 1657]),
    (1, 4, [300, 1], [4000, 4000]),
    (1, 8, [300], [2000]),
])
def test_every_partial_that_is_folded_has_been_written(Hkv, G, seqs, lens):
    p = _packed(torch.bfloat16, Hkv, G, 16, seqs, lens, room=int(4.6e6 / ((sum(seqs) - len(seqs)) * Hkv * G)))
    check_against(_run(p, 128 ** -0.5), _oracle(p, 128 ** -0.5).numpy(), torch.bfloat16)


def test_rows_that_nobody_sees_never_reach_a_result():
    """A sequence that already holds keys behind the ones this call's tokens may see."""
    p = _packed(torch.bfloat16, 2, 4, 16, [130, 1], [700, 300], room=5000)
    p["locations"] = (p["locations"] - 100).contiguous()
    ref = _oracle(p, 128 ** -0.5)
    for w, n in enumerate((600, 200)):
        for x in range(n, 16 * (n // 16 + 6)):
            p["value_cache"][p["block_table"][w, x // 16], :, x % 16] = float("nan")
    check_against(_run(p, 128 ** -0.5), ref.numpy(), torch.bfloat16)


@pytest.mark.parametrize("scale", [0.0, -0.05, 1e-40])
def test_scales_that_are_not_positive(scale):
    """The result for -scale is that of the negated queries for scale; a scale of nothing is an average over what a token sees.
    (The oracle masks before it scales and cannot say either by itself.)"""
    p = _packed(torch.bfloat16, 2, 4, 16, [200, 1], [700, 650], room=5000)
    flipped = dict(p, queries=-p["queries"] if scale < -0.01 else torch.zeros_like(p["queries"]))
    check_against(_run(p, scale), _oracle(flipped, max(0.01, -scale)).numpy(), torch.bfloat16)


SWITCH = """
from inference_lib_b200 import _cabi
p = _cabi.PagedProblem()
p.F, p.W, p.Hq, p.Hkv, p.E, p.Ev, p.dtype, p.cu_seqlens_q = 1, 4, 16, 4, 128, 128, _cabi.BF16, 1
p.total_q_tokens, p.num_blocks, p.block_size, p.max_blocks_per_seq = 300, 256, 16, 64
needs = []
for p.kernel in (_cabi.KERNEL_AUTO, _cabi.KERNEL_FMA):
    needs.append(_cabi.load().hogatt_paged_workspace_bytes(p))
print("SAME" if needs[0] == needs[1] else "OTHER")
"""


@pytest.mark.parametrize("env,route", [({}, "OTHER"), ({"HOGATT_PAGED_MMA": "0"}, "SAME"), ({"HOGATT_DENSE": "0"}, "SAME")])
def test_switches_keep_auto_off_it(env, route):
    root = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))
    res = subprocess.run([sys.executable, "-c", SWITCH], env=dict(os.environ, **env), capture_output=True, text=True, timeout=300, cwd=root)
    assert res.returncode == 0 and res.stdout.split() == [route], res.stdout + res.stderr[-2000:]


def test_the_extent_of_caches_of_different_sizes():
    """A tensor map must not reach past the smaller cache."""
    p = {k: v.to(DEV) for k, v in _packed(torch.bfloat16, 2, 4, 16, [130, 1], [300, 300], room=5000).items()}
    for name in ("key_cache", "value_cache"):
        q = dict(p, **{name: torch.cat([p[name], p[name][:3]])})
        problem, _ = _cabi.bind_paged(out=torch.empty(131, 8, 128, dtype=torch.bfloat16, device=DEV), scale=0.1, **q)
        assert problem.num_blocks == min(q["key_cache"].shape[0], q["value_cache"].shape[0])
