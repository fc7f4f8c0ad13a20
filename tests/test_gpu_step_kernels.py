"""The kernels of a decode step around the attention op at the edges of their ranges: workers' orders longer than one pass of
a warp, sources with few or no real rows, several sources of one fragment, launches that follow one another without a pause."""
import numpy as np
import pytest
import torch

from inference_lib_b200 import _cabi
from oracle import hogwild_cache_oracle as oc

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _stream():
    return torch.cuda.current_stream().cuda_stream


@pytest.mark.parametrize("F", [1, 2, 31, 32, 33, 64, 65, 127, 128])
def test_step_metadata_for_orders_of_any_length(F):
    rng = np.random.default_rng(F)
    W, S = 5, 3
    order = np.full((W, F), -1, dtype=np.int32)
    for w in range(W):
        n = F if w == 0 else (0 if w == 1 else int(rng.integers(1, F + 1)))       # all fragments, none, some
        order[w, :n] = rng.permutation(F)[:n]
    lengths = rng.integers(S, 400, F).astype(np.int32)
    inv = (1.0 / (1e4 ** (np.arange(0, 8, 2) / 8))).astype(np.float32)
    loc = torch.full((F, W, S), -7, dtype=torch.int32, device=DEV)
    cos = torch.full((F, W, S, 8), float("nan"), dtype=torch.float32, device=DEV)
    sin = torch.full_like(cos, float("nan"))
    assert _cabi.step_plan(order=torch.from_numpy(order).to(DEV), fragment_lengths=torch.from_numpy(lengths).to(DEV),
                           inv_freq=torch.from_numpy(inv).to(DEV), S=S, locations=loc, cosines=cos, sines=sin,
                           round_tables_to=_cabi.F32, stream=_stream()) == 0
    want = oc.step_locations(order, lengths, S)
    assert np.array_equal(loc.cpu().numpy(), want)
    wc, ws = oc.rotary_tables(want, inv)
    # one unit in the last place of a value below 1, on either side
    assert (cos.cpu() - wc).abs().max() <= 2.5e-7 and (sin.cpu() - ws).abs().max() <= 2.5e-7


@pytest.mark.parametrize("dtype,E", [(torch.bfloat16, 128), (torch.float16, 72), (torch.float32, 64)])
@pytest.mark.parametrize("S", [1, 7, 130])
def test_appends_in_a_row(dtype, E, S):
    """Two appends and the step metadata after them, enqueued back to back: worker 1 has no real rows, worker 2 some, workers 0
    and 3 share a fragment, and the second append starts where the first one ended."""
    g = torch.Generator().manual_seed(S)
    W, Hkv, cap, write_to, rows = 4, 3, 4 * S + 40, [0, 1, 2, 0], [S, 0, (S + 1) // 2, S]
    starts = torch.tensor([5, 0, 11], dtype=torch.int32)
    inv = 1.0 / (1e4 ** (torch.arange(0, E, 2, dtype=torch.float32) / E))
    ks = [torch.full((Hkv, cap, E), 7.0, dtype=dtype, device=DEV) for _ in range(3)]
    vs = [torch.full((Hkv, cap, E), 7.0, dtype=dtype, device=DEV) for _ in range(3)]
    lens = [starts.to(DEV), torch.zeros(3, dtype=torch.int32, device=DEV), torch.zeros(3, dtype=torch.int32, device=DEV)]
    want_k = [torch.full((Hkv, 0, E), 0.0, dtype=dtype) for _ in range(3)]
    want_v = [torch.full((Hkv, 0, E), 0.0, dtype=dtype) for _ in range(3)]
    status, new_rows, inputs = torch.zeros(1, dtype=torch.int32, device=DEV), torch.tensor(rows, dtype=torch.int32, device=DEV), []
    for step in range(2):
        k, v = (torch.randn(W, Hkv, S, E, generator=g).to(dtype) for _ in range(2))
        cos, sin = oc.rotary_tables(torch.randint(0, 5000, (W, S), generator=g).numpy(), inv.numpy())
        rotated = oc.rotate_keys(k, cos, sin)
        for w in range(W):
            want_k[write_to[w]], want_v[write_to[w]] = oc.append(want_k[write_to[w]], want_v[write_to[w]], rotated[w], v[w], rows[w])
        inputs.append([t.to(DEV) for t in (k, v, cos, sin)])
    order = torch.tensor([[0, 1, 2], [2, 1, 0], [1, 0, 2], [2, -1, -1]], dtype=torch.int32, device=DEV)
    loc = torch.empty((3, W, S), dtype=torch.int32, device=DEV)
    tables = [torch.empty((3, W, S, E), dtype=torch.float32, device=DEV) for _ in range(2)]
    inv_dev = inv.to(DEV)
    torch.cuda.synchronize()
    for step, (k, v, cos, sin) in enumerate(inputs):
        assert _cabi.append(keys=k, values=v, cosines=cos, sines=sin, write_to=write_to, key_fragments=ks, value_fragments=vs,
                            lengths_in=lens[step], lengths_out=lens[step + 1], new_rows=new_rows, status=status, stream=_stream()) == 0
    assert _cabi.step_plan(order=order, fragment_lengths=lens[2], inv_freq=inv_dev, S=S, locations=loc, cosines=tables[0], sines=tables[1],
                           round_tables_to=_cabi.F32, stream=_stream()) == 0
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    total = [int(starts[f]) + want_k[f].shape[1] for f in range(3)]
    assert lens[2].tolist() == total
    assert np.array_equal(loc.cpu().numpy(), oc.step_locations(order.cpu().numpy(), total, S))
    for f in range(3):
        a, b = int(starts[f]), total[f]
        assert torch.equal(ks[f][:, a:b].cpu(), want_k[f]) and torch.equal(vs[f][:, a:b].cpu(), want_v[f])
        for slab in (ks[f], vs[f]):
            assert (slab[:, :a] == 7).all() and (slab[:, b:] == 7).all()


@pytest.mark.parametrize("dtype,E,rows", [(torch.bfloat16, 128, (592, 593, 2000)), (torch.float16, 64, (1184, 1185)), (torch.float32, 128, (74, 75))])
def test_appends_of_a_prompts_rows(dtype, E, rows):
    """Around four CTAs per SM (of 148): few rows' CTAs hold more registers."""
    g = torch.Generator().manual_seed(E)
    Hkv, inv = 8, 1.0 / (1e4 ** (torch.arange(0, E, 2, dtype=torch.float32) / E))
    for S in rows:
        k, v = (torch.randn(1, Hkv, S, E, generator=g).to(dtype) for _ in range(2))
        cos, sin = oc.rotary_tables(torch.arange(3, 3 + S)[None].numpy(), inv.numpy())
        kf, vf = (torch.full((Hkv, S + 9, E), 7.0, dtype=dtype, device=DEV) for _ in range(2))
        lens = [torch.tensor([3], dtype=torch.int32, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)]
        d = [t.to(DEV) for t in (k, v, cos, sin)]
        assert _cabi.append(keys=d[0], values=d[1], cosines=d[2], sines=d[3], write_to=[0], key_fragments=[kf], value_fragments=[vf],
                            lengths_in=lens[0], lengths_out=lens[1], stream=_stream()) == 0
        torch.cuda.synchronize()
        assert lens[1].tolist() == [3 + S]
        assert torch.equal(kf[:, 3:3 + S].cpu(), oc.rotate_keys(k, cos, sin)[0]) and torch.equal(vf[:, 3:3 + S].cpu(), v[0])
        for slab in (kf, vf):
            assert (slab[:, :3] == 7).all() and (slab[:, 3 + S:] == 7).all()
