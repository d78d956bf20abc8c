"""GPU parity, routing: expert indices bit-exact against the oracle (both its operator form and the CPU daemon's form),
weights bit-exact against the operator form and within 2 ulp of the daemon's division form."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def E():
    import eke_hive_b200 as E
    return E


@pytest.mark.parametrize("M,Ex,k,renorm,lbf", [(1, 64, 8, True, True), (16, 512, 10, True, True), (33, 160, 8, False, True),
                                              (7, 1024, 16, True, False), (5, 37, 3, True, False)])
def test_softmax_router_bit_exact(E, oracle, M, Ex, k, renorm, lbf):
    import torch
    rng = np.random.default_rng(M * 1000 + Ex + k)
    lg = rng.normal(0, 1, (M, Ex + 3)).astype(np.float32)        # ld > E: trailing columns are not router logits
    ids, w = E.router_softmax_topk(torch.from_numpy(lg).cuda(), k, renorm, lbf, E=Ex)
    i0, w0 = oracle.router_softmax_topk(lg, k, renorm, lbf, 0, E=Ex)
    assert np.array_equal(ids.cpu().numpy(), i0)
    assert w.cpu().numpy().tobytes() == w0.tobytes()
    i1, w1 = oracle.router_softmax_topk(lg, k, renorm, lbf, 1, E=Ex)
    assert np.array_equal(ids.cpu().numpy(), i1)
    assert np.max(np.abs(w.cpu().numpy() - w1) / w1) < 1e-6


def test_softmax_router_ties(E, oracle):
    import torch
    lg = np.array([[1.0, 3.0, 3.0, -2.0, 3.0, 0.5, 3.0009765625, 1.0], [0.0] * 8], np.float32)
    ids, w = E.router_softmax_topk(torch.from_numpy(lg).cuda(), 3, True, True)
    assert ids.cpu().numpy().tolist() == [[1, 2, 4], [0, 1, 2]]
    ids, _ = E.router_softmax_topk(torch.from_numpy(lg).cuda(), 3, True, False)
    assert ids.cpu().numpy().tolist() == [[6, 1, 2], [0, 1, 2]]
    # bf16-rounded logits make ties common: a whole batch must still agree with the oracle
    rng = np.random.default_rng(11)
    lg = np.round(rng.normal(0, 1, (64, 512)) * 4).astype(np.float32) / 4
    ids, w = E.router_softmax_topk(torch.from_numpy(lg).cuda(), 10, True, True)
    i0, w0 = oracle.router_softmax_topk(lg, 10, True, True, 0)
    assert np.array_equal(ids.cpu().numpy(), i0) and w.cpu().numpy().tobytes() == w0.tobytes()


@pytest.mark.parametrize("M,Ex,k", [(8, 160, 8), (1, 256, 8), (19, 64, 6)])
def test_sigmoid_router_bit_exact(E, oracle, M, Ex, k):
    import torch
    rng = np.random.default_rng(M + Ex)
    lg = rng.normal(0, 1, (M, Ex)).astype(np.float32)
    bias = rng.normal(0, 0.3, Ex).astype(np.float32)
    ids, w = E.router_topk(torch.from_numpy(lg).cuda(), torch.from_numpy(bias).cuda(), k, 2.5)
    i0, w0 = oracle.router_sigmoid_topk(lg, bias, k, 2.5, 0)
    assert np.array_equal(ids.cpu().numpy(), i0) and w.cpu().numpy().tobytes() == w0.tobytes()
    i1, w1 = oracle.router_sigmoid_topk(lg, bias, k, 2.5, 1)
    assert np.array_equal(ids.cpu().numpy(), i1)
    assert np.max(np.abs(w.cpu().numpy() - w1) / w1) < 1e-6
    ids, w = E.router_topk(torch.from_numpy(lg).cuda(), None, k, 1.0)
    i0, w0 = oracle.router_sigmoid_topk(lg, None, k, 1.0, 0)
    assert np.array_equal(ids.cpu().numpy(), i0) and w.cpu().numpy().tobytes() == w0.tobytes()


def test_zipf_biased_routing_matches(E, oracle):
    """Hot-expert skew (N(0,1) logits plus a per-expert Zipf(1.1) log-weight bias): indices still bit-exact."""
    import torch
    rng = np.random.default_rng(12)
    Ex = 160
    zipf = 1.0 / np.arange(1, Ex + 1) ** 1.1
    bias = np.log(zipf / zipf.sum())[rng.permutation(Ex)].astype(np.float32)
    lg = (rng.normal(0, 1, (8, Ex)) + bias).astype(np.float32)
    ids, w = E.router_softmax_topk(torch.from_numpy(lg).cuda(), 8, True, True)
    i0, w0 = oracle.router_softmax_topk(lg, 8, True, True, 0)
    assert np.array_equal(ids.cpu().numpy(), i0) and w.cpu().numpy().tobytes() == w0.tobytes()


@pytest.mark.parametrize("Ex", [16, 31, 255, 256, 257, 511, 512, 513, 1023, 1024])
def test_router_register_widths(E, oracle, Ex):
    """The stand-alone routers (one warp a row) at the edges of a lane's share of the experts, with whole groups of equal scores: ids and
    weights are integers and fp32 results of the same operations in the same order, so they are compared bit for bit."""
    import torch
    rng = np.random.default_rng(Ex)
    k = 16
    lg = (np.round(rng.normal(0, 1, (9, Ex)) * 4) / 4).astype(np.float32)
    lg[1] = 0.25                                                  # all equal: the first k ids
    lg[2] = -np.inf; lg[2, Ex // 2] = 1.0                         # one score far above the others, which all clamp to the same exp
    for renorm in (True, False):
        ids, w = E.router_softmax_topk(torch.from_numpy(lg).cuda(), k, renorm, False)
        i0, w0 = oracle.router_softmax_topk(lg, k, renorm, False, 0)
        assert np.array_equal(ids.cpu().numpy(), i0) and w.cpu().numpy().tobytes() == w0.tobytes()
    lg[2] = 0.5
    bias = (np.round(rng.normal(0, 1, Ex) * 2) / 2).astype(np.float32)     # negative sums of score and bias among them
    for b in (bias, None):
        ids, w = E.router_topk(torch.from_numpy(lg).cuda(), None if b is None else torch.from_numpy(b).cuda(), k, 2.5)
        i0, w0 = oracle.router_sigmoid_topk(lg, b, k, 2.5, 0)
        assert np.array_equal(ids.cpu().numpy(), i0) and w.cpu().numpy().tobytes() == w0.tobytes()


@pytest.mark.parametrize("kind", ["softmax", "sigmoid"])
@pytest.mark.parametrize("Ex", [16, 31, 512, 1024])
def test_layer_routing_at_every_group_width(E, oracle, kind, Ex):
    """The routing inside the decode layer's grouping kernel: one CTA with 16 and 8 warps a row (1 and 2 rows), a cluster with 16, 8, 4 and 2 warps a
    row (3-8, 9-16, 17-32, 33-64 rows; the last of each range leaves groups without a row).  Rows of equal scores and rows with one score above
    all others have more than 64 candidates wherever there are that many experts.  Ids and weights bit for bit against the oracle."""
    import torch

    from util import bf16_tensor, random_records, upload
    H, I, k = 256, 256, 16
    keep = upload(random_records(oracle, H, I, 4, Ex))
    tab = E.rec_table([keep[e % 3] for e in range(Ex)])
    for M in (1, 2, 3, 8, 9, 16, 17, 32, 33, 45, 64):
        rng = np.random.default_rng(1000 * M + Ex)
        lg = rng.normal(0, 1, (M, Ex)).astype(np.float32)
        lg[::2] = np.round(lg[::2] * 4) / 4                       # runs of equal scores
        special = M - 1 if M < 9 else M - 2
        lg[special] = 0.25                                        # all equal: the first k ids
        if M > 2:
            lg[1] = -np.inf if kind == "softmax" else -3.0
            lg[1, Ex // 2] = 1.0                                  # one far above the others, which are equal
        x = bf16_tensor(oracle.bf16r(rng.normal(0, 1, (M, H)).astype(np.float32)))
        for variant in (0, 1):
            if kind == "softmax":
                ids, w, _ = E.moe_layer_decode(torch.from_numpy(lg).cuda(), x, tab, 0, Ex, k, H, I, shared_rec=keep[3], renorm=variant == 0, logits_bf16=variant == 0)
                i0, w0 = oracle.router_softmax_topk(lg, k, variant == 0, variant == 0, 0)
            else:
                bias = None if variant else (np.round(rng.normal(0, 1, Ex) * 2) / 2).astype(np.float32)
                ids, w, _ = E.moe_layer_decode(torch.from_numpy(lg).cuda(), x, tab, 0, Ex, k, H, I, shared_rec=keep[3],
                                               bias=None if bias is None else torch.from_numpy(bias).cuda(), sigmoid_scale=2.5)
                i0, w0 = oracle.router_sigmoid_topk(lg, bias, k, 2.5, 0)
            assert np.array_equal(ids.cpu().numpy(), i0), (M, variant)
            assert w.cpu().numpy().tobytes() == w0.tobytes(), (M, variant)
    E.context().check_device()


@pytest.mark.parametrize("Ex,k", [(1, 1), (2, 1), (7, 7), (8, 3), (32, 1), (32, 16), (33, 16)])
def test_routers_of_few_experts(E, oracle, Ex, k):
    """Up to 32 experts a row sits in the lanes of a warp: equal scores, one finite score, every expert picked, logits rows longer than E; one
    expert more takes the general way."""
    import torch
    rng = np.random.default_rng(100 * Ex + k)
    lg = (np.round(rng.normal(0, 1, (11, Ex + 2)) * 4) / 4).astype(np.float32)
    lg[1] = 0.25
    lg[2] = -np.inf; lg[2, Ex // 2] = 1.0
    lg[3] = rng.normal(0, 30, Ex + 2)                            # scores that underflow beside the largest
    for renorm, lbf in ((True, True), (False, False)):
        ids, w = E.router_softmax_topk(torch.from_numpy(lg).cuda(), k, renorm, lbf, E=Ex)
        i0, w0 = oracle.router_softmax_topk(lg, k, renorm, lbf, 0, E=Ex)
        assert np.array_equal(ids.cpu().numpy(), i0) and w.cpu().numpy().tobytes() == w0.tobytes()
    ls = np.ascontiguousarray(lg[:, :Ex])
    ls[2] = 0.5
    bias = (np.round(rng.normal(0, 1, Ex) * 2) / 2).astype(np.float32)
    for b in (bias, None):
        ids, w = E.router_topk(torch.from_numpy(ls).cuda(), None if b is None else torch.from_numpy(b).cuda(), k, 2.5)
        i0, w0 = oracle.router_sigmoid_topk(ls, b, k, 2.5, 0)
        assert np.array_equal(ids.cpu().numpy(), i0) and w.cpu().numpy().tobytes() == w0.tobytes()


@pytest.mark.parametrize("B", [1, 2, 3, 4, 5, 33, 700])
def test_route_and_push_of_one_rank(E, oracle, B):
    """The expert-parallel route + push kernel with a single rank (nothing to wait for): 16, 8, 4 and 2 warps a row, and the most rows its
    shared memory takes (700 rows of 8 picks beside 16 experts' scores).  Rows, ids and weights arrive as the router gives them."""
    import torch
    H, Ex, k = 64, 16 if B == 700 else 160, 8
    rng = np.random.default_rng(B)
    lg = rng.normal(0, 1, (B, Ex)).astype(np.float32)
    lg[-1] = 0.5
    x = torch.from_numpy(rng.normal(0, 1, (B, H)).astype(np.float32)).bfloat16().cuda()
    mine = torch.zeros(E.PeerExchange.layout(1, B, H, k)[1], dtype=torch.uint8, device="cuda")
    ex = E.PeerExchange(mine, lambda o: [o], 0, 1, B, H, k)
    ids, w = torch.zeros((B, k), dtype=torch.int32, device="cuda"), torch.zeros((B, k), device="cuda")
    ex.route_push(torch.from_numpy(lg).cuda(), x, ids, w, Ex)
    torch.cuda.synchronize()
    i0, w0 = oracle.router_softmax_topk(lg, k, True, True, 0)
    assert np.array_equal(ids.cpu().numpy(), i0) and w.cpu().numpy().tobytes() == w0.tobytes()
    rec = mine[ex.off["recv"]:ex.off["recv"] + B * ex.rec_bytes].reshape(B, ex.rec_bytes)
    assert torch.equal(rec[:, :2 * H].contiguous().view(torch.int16), x.view(torch.int16))
    assert torch.equal(rec[:, 2 * H:2 * H + 4 * k].contiguous().view(torch.int32), ids)
    assert torch.equal(rec[:, 2 * H + 4 * k:2 * H + 8 * k].contiguous().view(torch.float32), w)
    E.context().check_device()
    ex.close()
