"""Attention with a sink and a bias by distance in steps of many tokens: the bits of its results.

Where a cap and the bias of the table's last column meet, the constant that both add to a score is rounded once, as
cap log2(e) + bias in one multiply-add; a second rounding moves the weights of all keys beyond the table by about 2^-18, which
routers behind the layer turn into other experts.  The digests are those of the kernel from before its masks and biases moved
behind branches of their own."""
import hashlib

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def outputs(split, cap, table_len, window):
    from mivi_v4_b200.ops import kernels as K
    lens, starts, nh, nkv, dk, dv, page = [150, 333], [40, 0], 4, 2, 64, 64, 64
    g = torch.Generator().manual_seed(3)
    blocks = [-(-(n + s) // page) for n, s in zip(lens, starts)]
    pool = torch.randn(sum(blocks), nkv * page * (dk + dv), generator=g).to(torch.bfloat16)
    table = torch.zeros(len(lens), max(blocks), dtype=torch.int32)
    for b, n in enumerate(blocks):
        table[b, :n] = torch.arange(n) + sum(blocks[:b])
    q = torch.randn(sum(lens), nh * dk, generator=g).to(torch.bfloat16)
    bias = torch.randn(nh, table_len, generator=g)
    out = torch.zeros(sum(lens), nh * dv, dtype=torch.bfloat16, device=DEV)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)     # noqa: E731
    K.attention_sink_prefill(q.to(DEV), pool.to(DEV), page, table.to(DEV), i32([0, 150, 483]), i32(starts), out, 2, nh, nkv, dk, dv,
                             0.125, softcap=cap, window=window, distance_table=bias.to(DEV), split_weights=split)
    return out.cpu()


def digest(t):
    return hashlib.sha256(t.view(torch.int16).numpy().tobytes()).hexdigest()[:16]


GOLDEN = {(True, 50.0, 16, 0): "91c2f49550306ab7", (False, 50.0, 16, 0): "31251ef446f0f1dd",
          (True, 7.0, 64, 100): "8e790072657b02ae", (True, 0.0, 16, 0): "c4ef7403df5f2677"}


@pytest.mark.parametrize("split,cap,table_len,window", list(GOLDEN))
def test_a_cap_and_the_last_distance_are_rounded_once(split, cap, table_len, window):
    assert digest(outputs(split, cap, table_len, window)) == GOLDEN[split, cap, table_len, window]
