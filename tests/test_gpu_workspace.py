"""A call stays inside the workspace whose size its *_ws_bytes function gives: the workspace is the front of a larger buffer, and the
rest of that buffer is the same bytes before and after."""
import numpy as np
import pytest
import torch

from util import random_records, upload

pytestmark = pytest.mark.gpu

GUARD = 32 << 20                                                         # more than any operator's scratch at the sizes below


@pytest.fixture(scope="module")
def E():
    import eke_hive_b200 as E
    return E


def guarded(nbytes):
    buf = torch.full((nbytes + GUARD,), 0xA5, dtype=torch.uint8, device="cuda")
    return buf[:nbytes], buf[nbytes:]


def untouched(tail):
    torch.cuda.synchronize()
    return bool((tail == 0xA5).all())


@pytest.mark.parametrize("M", [65, 100, 129])
def test_layer_beyond_64_rows_without_a_grouped_gemm(E, oracle, M):
    """Decode calls of 64 rows, on the tensor-memory gate/up kernel (its digit planes are the largest part of the scratch)."""
    H, I, E_, K = 2048, 512, 16, 8
    keep = upload(random_records(oracle, H, I, E_ + 1, M))
    tab = E.rec_table(keep[:E_])
    g = torch.Generator().manual_seed(M)
    x = torch.randn((M, H), generator=g).bfloat16().cuda()
    lg = torch.randn((M, E_ + 1), generator=g).cuda()
    ws, tail = guarded(E.moe_layer_ws_bytes(M, K, E_, H, I))
    ids, w, out = E.moe_layer(lg, x, tab, 0, E_, K, H, I, shared_rec=keep[E_], gate_col=E_, ws=ws)
    assert untouched(tail)
    for m0 in range(0, M, 64):
        sl = slice(m0, min(M, m0 + 64))
        ref = E.moe_layer_decode(lg[sl], x[sl], tab, 0, E_, K, H, I, shared_rec=keep[E_], gate_col=E_)
        assert torch.equal(out[sl].view(torch.int16), ref[2].view(torch.int16)) and torch.equal(ids[sl], ref[0])
    E.context().check_device()


@pytest.mark.parametrize("M,S,K,E_", [(16, 1, 1, 1), (20, 1, 2, 3), (33, 3, 1, 1)])
def test_prefill_few_rows_in_small_slices(E, oracle, M, S, K, E_):
    """bf16 activations, few rows, slices of a row or three: the workspace of such a slice is too small for the tensor-memory kernel's digit
    planes, which a call of so many pairs would use."""
    H, I = 2048, 512
    tab = E.rec_table(keep := upload(random_records(oracle, H, I, E_, M)))
    g = torch.Generator().manual_seed(M)
    x = torch.randn((M, H), generator=g).bfloat16().cuda()
    ids = torch.stack([torch.randperm(E_, generator=g)[:K] for _ in range(M)]).int().cuda()
    w = torch.rand((M, K), generator=g).cuda()
    ctx, pinned = E.Context(flags=E.HB_FLAG_PREFILL_A16), E.Context(flags=E.HB_FLAG_DECODE_MMA_SYNC)
    ws, tail = guarded(E.moe_prefill_ws_bytes(S, K, E_, H, I))
    out = E.fn_moe_prefill(tab, 0, E_, ids, w, x, H, I, ws=ws, S=S, ctx=ctx)
    assert untouched(tail)
    ref = E.moe_decode_routed_f32(ids, w, tab, 0, E_, x, H, I, ctx=pinned)
    rms = ref.double().pow(2).mean(1, keepdim=True).sqrt()
    assert float(((out.double() - ref.double()).abs() / rms).max()) <= 2e-2     # the gate of the decode operators, whichever engine a slice gets
    ctx.check_device(); pinned.check_device()
    ctx.close(); pinned.close()
    del keep
