"""The operators either side of the attention op (``fragment_append``, ``fragment_step_plan``): what does not fit together is
refused on the host, before anything is launched, and the forms they take give what the C ABI gives."""
import pytest
import torch

from inference_lib_b200 import _cabi
import inference_lib_b200.attention as A

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
W, Hkv, S, E, Ev, F, CAP = 2, 3, 4, 32, 16, 3, 24


def _append_args(dtype=torch.bfloat16):
    g = torch.Generator().manual_seed(0)
    angle = torch.rand(W, S, E, generator=g)
    return dict(keys=torch.randn(W, Hkv, S, E, generator=g).to(DEV, dtype), values=torch.randn(W, Hkv, S, Ev, generator=g).to(DEV, dtype),
                cosines=angle.cos().to(DEV), sines=angle.sin().to(DEV), write_to=[1, 2],
                key_fragments=[torch.zeros(Hkv, CAP, E, dtype=dtype, device=DEV) for _ in range(F)],
                value_fragments=[torch.zeros(Hkv, CAP, Ev, dtype=dtype, device=DEV) for _ in range(F)],
                lengths_in=torch.tensor([5, 0, 3], dtype=torch.int32, device=DEV), lengths_out=torch.zeros(F, dtype=torch.int32, device=DEV),
                new_rows=torch.tensor([S, 2], dtype=torch.int32, device=DEV), take_leading=False,
                status=torch.zeros(1, dtype=torch.int32, device=DEV))


def _change_one(name, i, fn):
    return lambda a: a[name].__setitem__(i, fn(a[name][i]))


def _change(name, fn):
    return lambda a: a.__setitem__(name, fn(a[name]))


REFUSED = {
    "cosines on the host": _change("cosines", lambda t: t.cpu()),
    "new_rows on the host": _change("new_rows", lambda t: t.cpu()),
    "lengths on the host": _change("lengths_in", lambda t: t.cpu()),
    "lengths_out on the host": _change("lengths_out", lambda t: t.cpu()),
    "status on the host": _change("status", lambda t: t.cpu()),
    "a key fragment on the host": _change_one("key_fragments", 0, lambda t: t.cpu()),
    "a value fragment on the host": _change_one("value_fragments", 2, lambda t: t.cpu()),
    "values on the host": _change("values", lambda t: t.cpu()),
    "values of another type": _change("values", lambda t: t.half()),
    "a key fragment of another type": _change_one("key_fragments", 1, lambda t: t.float()),
    "a value fragment of another type": _change_one("value_fragments", 1, lambda t: t.half()),
    "sines of another type": _change("sines", lambda t: t.bfloat16()),
    "tables of a third type": lambda a: a.update(cosines=a["cosines"].half(), sines=a["sines"].half()),
    "new_rows of 64 bits": _change("new_rows", lambda t: t.long()),
    "lengths of 64 bits": _change("lengths_in", lambda t: t.long()),
    "status of 64 bits": _change("status", lambda t: t.long()),
    "values of fewer sources": _change("values", lambda t: t[:1]),
    "values of fewer heads": _change("values", lambda t: t[:, :2]),
    "values of fewer rows": _change("values", lambda t: t[:, :, :2]),
    "values of another head size": _change("values", lambda t: torch.cat([t, t], -1)),
    "sines of fewer rows": _change("sines", lambda t: t[:, :2]),
    "sines of a shorter row": _change("sines", lambda t: t[..., :16]),
    "one row of cosines, two of sines": lambda a: a.update(cosines=a["cosines"][:1, :1], sines=a["sines"][:1, :2]),
    "new_rows of fewer sources": _change("new_rows", lambda t: t[:1]),
    "lengths of fewer fragments": _change("lengths_in", lambda t: t[:2]),
    "lengths_out of fewer fragments": _change("lengths_out", lambda t: t[:2]),
    "lengths that are one and the same": lambda a: a.update(lengths_out=a["lengths_in"]),
    "no status": _change("status", lambda t: t[:0]),
    "a fragment of fewer heads": _change_one("key_fragments", 0, lambda t: t[:2]),
    "a fragment of another head size": _change_one("key_fragments", 0, lambda t: t.view(Hkv, CAP * 2, E // 2)),
    "a value fragment of fewer rows": _change_one("value_fragments", 1, lambda t: t[:, :8].contiguous()),
    "a value fragment of another head size": _change_one("value_fragments", 1, lambda t: t.view(Hkv, CAP // 2, Ev * 2)),
    "a fragment with gaps": _change_one("key_fragments", 1, lambda t: t[:, :8]),
    "fewer value fragments": _change("value_fragments", lambda t: t[:2]),
    "a fragment that is not there": _change("write_to", lambda t: [1, 3]),
    "a fragment that is not there, 2^32 later": _change("write_to", lambda t: [1, 1 << 32]),
    "a negative fragment": _change("write_to", lambda t: [1, -1]),
    "one target for two sources": _change("write_to", lambda t: [1]),
    "keys without a contiguous last axis": _change("keys", lambda t: torch.cat([t, t], -1)[..., ::2]),
    "keys of three axes": _change("keys", lambda t: t[0]),
}


@pytest.mark.parametrize("what", list(REFUSED))
def test_appends_that_are_refused(what):
    a = _append_args()
    REFUSED[what](a)
    with pytest.raises((RuntimeError, IndexError)):
        A.fragment_append(*a.values())
    torch.cuda.synchronize()
    assert all(not t.any() for t in a["key_fragments"] + a["value_fragments"])


def _views(a):
    """Sources as transposed views of a projection's output, slabs with a leading 1."""
    for k in ("keys", "values"):
        a[k] = a[k].transpose(1, 2).contiguous().transpose(1, 2)
    a["key_fragments"] = [t[None] for t in a["key_fragments"]]
    a["value_fragments"] = [t[None] for t in a["value_fragments"]]


ACCEPTED = {
    "as they are": lambda a: None,
    "views": _views,
    "one row of tables for all": lambda a: a.update(cosines=a["cosines"][0, 0], sines=a["sines"][:1, :1]),
    "rows shared by the workers": lambda a: a.update(cosines=a["cosines"][:1].expand(W, S, E), sines=a["sines"][:1].expand(W, S, E)),
    "tables of the model's type": lambda a: a.update(cosines=a["cosines"].bfloat16(), sines=a["sines"].bfloat16()),
    "part of the head rotated": lambda a: a.update(cosines=a["cosines"][..., :16], sines=a["sines"][..., :16]),
    "all rows": lambda a: a.update(new_rows=None),
    "leading rows": lambda a: a.update(take_leading=True),
}


@pytest.mark.parametrize("what", list(ACCEPTED))
def test_appends_that_are_taken(what):
    got, want = _append_args(), _append_args()
    ACCEPTED[what](got)
    ACCEPTED[what](want)
    A.fragment_append(*got.values())
    assert _cabi.append(stream=torch.cuda.current_stream().cuda_stream, **want) == 0
    torch.cuda.synchronize()
    assert got["key_fragments"][1].any() and got["lengths_out"].tolist() == want["lengths_out"].tolist()
    for name in ("key_fragments", "value_fragments"):
        for x, y in zip(got[name], want[name]):
            assert torch.equal(x, y)


def _plan_args():
    return dict(order=torch.tensor([[0, 2, 1], [0, 1, 2]], dtype=torch.int32, device=DEV), fragment_lengths=torch.tensor([9, 5, 6], dtype=torch.int32, device=DEV),
                inv_freq=torch.rand(E // 2, device=DEV), locations=torch.zeros(F, W, S, dtype=torch.int32, device=DEV),
                cosines=torch.zeros(F, W, S, E, device=DEV), sines=torch.zeros(F, W, S, E, device=DEV), attention_scaling=1.0,
                round_tables_to=_cabi.F32)


PLANS_REFUSED = {
    "lengths on the host": _change("fragment_lengths", lambda t: t.cpu()),
    "frequencies on the host": _change("inv_freq", lambda t: t.cpu()),
    "tables on the host": _change("sines", lambda t: t.cpu()),
    "an order of 64 bits": _change("order", lambda t: t.long()),
    "lengths of 64 bits": _change("fragment_lengths", lambda t: t.long()),
    "frequencies of 64 bits": _change("inv_freq", lambda t: t.double()),
    "tables of 16 bits": _change("cosines", lambda t: t.bfloat16()),
    "lengths of fewer fragments": _change("fragment_lengths", lambda t: t[:2]),
    "locations of fewer fragments": _change("locations", lambda t: t[:2]),
    "locations of fewer workers": _change("locations", lambda t: t[:, :1].contiguous()),
    "locations of more rows than the tables": _change("locations", lambda t: torch.cat([t, t], 2)),
    "tables of fewer fragments": _change("cosines", lambda t: t[:2]),
    "tables of fewer workers": _change("sines", lambda t: t[:, :1].contiguous()),
    "shorter rows": _change("sines", lambda t: t[..., :16].contiguous()),
    "more frequencies than a row takes": _change("inv_freq", lambda t: torch.cat([t, t])),
    "tables with gaps": _change("cosines", lambda t: torch.cat([t, t], -1)[..., :E]),
    "an order with gaps": _change("order", lambda t: torch.cat([t, t], 1)[:, :F]),
}


@pytest.mark.parametrize("what", list(PLANS_REFUSED))
def test_step_metadata_that_is_refused(what):
    a = _plan_args()
    PLANS_REFUSED[what](a)
    with pytest.raises((RuntimeError, IndexError)):
        A.fragment_step_plan(*a.values())
    torch.cuda.synchronize()
    assert not a["cosines"].any() and not a["locations"].any()


def test_step_metadata_that_is_taken():
    got, want = _plan_args(), _plan_args()
    want["inv_freq"] = got["inv_freq"]
    A.fragment_step_plan(*got.values())
    assert _cabi.step_plan(S=S, stream=torch.cuda.current_stream().cuda_stream, **want) == 0
    torch.cuda.synchronize()
    assert got["locations"].any() and got["cosines"].any()
    for name in ("locations", "cosines", "sines"):
        assert torch.equal(got[name], want[name])
