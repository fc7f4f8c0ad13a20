"""Queries and keys that are not numbers: the rows they belong to are NaN -- not zero as for a row that sees nothing, and not a
mean over the keys that are left -- and no other row is."""
import pytest
import torch

from inference_lib_b200 import _cabi
from inference_lib_b200 import attention as ops
from inference_lib_b200 import workloads as wl
from tests.gpu_util import run_cabi

pytestmark = pytest.mark.gpu


def _problem(dtype, E, G, Hkv, S=1, lengths=(128, 270, 71)):
    return wl.make_problem("nan", W=2, Hq=Hkv * G, Hkv=Hkv, E=E, S=S, lengths=list(lengths), theta=5e5, dtype=dtype, seed=4)


CALLS = [
    (torch.float32, 64, 2, 2, 1, _cabi.KERNEL_AUTO),         # the fp32 kernel, 8 and 16 rows
    (torch.float32, 128, 8, 2, 1, _cabi.KERNEL_AUTO),
    (torch.float32, 32, 2, 2, 1, _cabi.KERNEL_AUTO),         # the kernel for other head sizes
    (torch.bfloat16, 128, 4, 2, 1, _cabi.KERNEL_MMA),
    (torch.float16, 64, 4, 1, 3, _cabi.KERNEL_MMA),          # one kv head: many partials
    (torch.bfloat16, 128, 4, 2, 1, _cabi.KERNEL_MMA_CLUSTER),
    (torch.bfloat16, 128, 4, 2, 32, _cabi.KERNEL_AUTO),      # the tcgen05 kernels
]


@pytest.mark.parametrize("dtype,E,G,Hkv,S,kernel", CALLS)
@pytest.mark.parametrize("max_ctas", [0, 2])
def test_a_query_that_is_not_a_number(dtype, E, G, Hkv, S, kernel, max_ctas):
    p = _problem(dtype, E, G, Hkv, S, lengths=(128, 270 + S, 71 + S))
    p.queries[1, 1, S - 1, 3] = float("nan")
    r = run_cabi(p, kernel=kernel, max_ctas=max_ctas)
    assert r.rc == 0 and r.status == 0
    rows = torch.isnan(r.out).all(-1).cpu()
    assert rows[1, 1, S - 1] and int(rows.sum()) == 1 and int(torch.isnan(r.out).sum()) == p.Ev


@pytest.mark.parametrize("dtype,E,G,Hkv,S,kernel", CALLS[:6])
@pytest.mark.parametrize("max_ctas", [0, 2])
def test_keys_that_are_not_numbers(dtype, E, G, Hkv, S, kernel, max_ctas):
    """A fragment of them in front of good ones, two whole tiles of the fp32 kernel; the second worker does not see it."""
    p = _problem(dtype, E, G, Hkv, S, lengths=(128, 270 + S, 71 + S))
    p.keys[0][:] = float("nan")
    loc = p.locations.clone()
    loc[0, 1] = -1
    r = run_cabi(wl.Problem(**{**p.__dict__, "locations": loc}), kernel=kernel, max_ctas=max_ctas)
    assert r.rc == 0 and r.status == 0
    assert torch.isnan(r.out[0]).all() and torch.isfinite(r.out[1]).all()


@pytest.mark.parametrize("E,block", [(128, 16), (128, 12), (64, 16)])
def test_paged(E, block):
    gen = torch.Generator(device="cuda").manual_seed(5)
    kc, vc = (torch.randn(30, 2, block, E, device="cuda", generator=gen).bfloat16() for _ in range(2))
    q = torch.randn(1, 2, 8, 1, E, device="cuda", generator=gen).bfloat16()
    q[0, 1, 2, 0, 5] = float("nan")
    table = torch.arange(30, dtype=torch.int32, device="cuda").reshape(2, 15)
    loc = torch.full((1, 2, 1), 140, dtype=torch.int32, device="cuda")
    out = ops.hogwild_paged_sdpa(q, loc, kc, vc, table, E ** -0.5, torch.tensor([141], dtype=torch.int32, device="cuda"))
    rows = torch.isnan(out).all(-1)
    assert bool(rows[1, 2, 0]) and int(rows.sum()) == 1 and int(torch.isnan(out).sum()) == E
