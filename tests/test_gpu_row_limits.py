"""Query rows of one block that see different numbers of keys (causal chunks), on the mma.sync kernel's 32- and 64-row
blocks: several m-tiles share every slice of a tile, and what one of them does not see another one still needs."""
import pytest
import torch

from inference_lib_b200 import _cabi
from inference_lib_b200 import workloads as wl
from oracle import hogwild_oracle as oracle
from tests.gpu_util import check_against, run_cabi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,S,lengths,kernel", [
    (1, 7, [700], _cabi.KERNEL_MMA),                        # 28 rows: one 32-row block
    (1, 600, [600], _cabi.KERNEL_MMA),                      # a causal prompt: 38 blocks of 64 rows, most tiles cut by the limit
    (2, 50, [300, 90, 130], _cabi.KERNEL_MMA),
    (2, 50, [300, 90, 130], _cabi.KERNEL_MMA_CLUSTER),
])
def test_rows_of_a_block_with_different_limits(W, S, lengths, kernel):
    orders = [[0]] if len(lengths) == 1 else None
    p = wl.make_problem("limits", W=W, Hq=8, Hkv=2, E=128, S=S, lengths=lengths, theta=5e5, dtype=torch.bfloat16, seed=5,
                        orders=orders)
    ref, _ = oracle.fused(p.queries, p.cos, p.sin, p.locations, p.keys, p.values, p.scale)
    for host_lengths in (None, "rows"):
        a = run_cabi(p, kernel=kernel, host_lengths=host_lengths)
        b = run_cabi(p, kernel=kernel, host_lengths=host_lengths)
        assert a.rc == 0 and a.status == 0
        # probabilities and outputs are rounded to bf16 (2^-9 each, relative to values of at most 4.5): well inside
        # the parity tolerance; the same call twice gives the same bits
        check_against(a.out, ref.numpy(), p.dtype, what=f"S={S} host {host_lengths}")
        assert torch.equal(a.out, b.out)
