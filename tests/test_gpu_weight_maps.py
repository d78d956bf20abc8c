"""The tensor maps through which the tensor-memory decode kernel and the bf16-activation GEMM read expert records belong to the call: captured
calls replay correctly whatever ran on the context since, and records may sit at any 16-byte aligned address, however far apart."""
import pytest
import torch

from util import random_records, upload

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def E():
    import eke_hive_b200 as E
    return E


class Layer:
    """One layer of random records with its inputs; call() runs it and leaves the result in .out."""

    def __init__(self, E, oracle, ctx, M, K, H, I, n=8, seed=1, layer=False):
        self.E, self.ctx, self.M, self.K, self.H, self.I, self.n, self.layer = E, ctx, M, K, H, I, n, layer
        self.recs = upload(random_records(oracle, H, I, n + 1, seed))
        self.tab = E.rec_table(self.recs[:n])
        g = torch.Generator().manual_seed(seed)
        self.x = torch.randn((M, H), generator=g).bfloat16().cuda()
        self.lg = torch.randn((M, n + 1), generator=g).cuda()
        self.ids = torch.zeros((M, K), dtype=torch.int32, device="cuda")
        self.w = torch.zeros((M, K), device="cuda")
        self.out = torch.zeros((M, H), dtype=torch.bfloat16, device="cuda")
        nb = E.moe_layer_ws_bytes(M, K, n, H, I) if layer else E.moe_decode_ws_bytes(M * (K + 1), H, I)
        self.ws = torch.empty(nb, dtype=torch.uint8, device="cuda")

    def call(self, ctx=None, tab=None, shared=None):
        f = self.E.moe_layer if self.layer else self.E.moe_layer_decode
        f(self.lg, self.x, self.tab if tab is None else tab, 0, self.n, self.K, self.H, self.I, shared_rec=self.recs[self.n] if shared is None else shared,
          gate_col=self.n, ids=self.ids, w=self.w, out=self.out, ws=self.ws, ctx=ctx or self.ctx)

    def result(self, **kw):
        self.out.zero_()
        self.call(**kw)
        torch.cuda.synchronize()
        return self.out.clone()

    def capture(self, warm):
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        if warm:
            with torch.cuda.stream(side):
                self.call()
            torch.cuda.current_stream().wait_stream(side)
        torch.cuda.synchronize()
        self.graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(self.graph):
            self.call()

    def replayed(self):
        self.out.zero_()
        self.graph.replay()
        torch.cuda.synchronize()
        return self.out.clone()


def same(a, b):
    return torch.equal(a.view(torch.int16), b.view(torch.int16))


@pytest.mark.parametrize("warm", [True, False])
def test_graphs_of_several_shapes_on_one_context(E, oracle, warm):
    """Captured decode calls of three shapes (all on the tensor-memory kernel: 9, 20 and 40 pairs) and a captured prefill layer, replayed after
    each other and after eager calls of further shapes; `warm` = False: the first call of a shape is made under capture."""
    ctx = E.Context(flags=E.HB_FLAG_PREFILL_A16)
    shapes = [(1, 8, 4096, 1536, False), (4, 4, 2048, 512, False), (8, 4, 1024, 512, False), (70, 4, 512, 256, True)]
    if not warm:                                                # module and kernel loading out of the way, on another context and shape
        other = E.Context(flags=E.HB_FLAG_PREFILL_A16)
        for M, layer in ((8, False), (70, True)):
            Layer(E, oracle, other, M, 4, 2048, 256, seed=7, layer=layer).result()
    layers = [Layer(E, oracle, ctx, M, K, H, I, seed=i + 1, layer=lay) for i, (M, K, H, I, lay) in enumerate(shapes)]
    for lay in layers:
        lay.capture(warm)
    fresh = E.Context(flags=E.HB_FLAG_PREFILL_A16)
    ref = [lay.result(ctx=fresh) for lay in layers]
    eager = Layer(E, oracle, ctx, 8, 4, 2048, 768, seed=9)
    eager_ref = eager.result(ctx=fresh)
    for order in ((0, 1, 2, 3), (3, 1, 0, 2)):
        for i in order:
            assert same(layers[i].replayed(), ref[i]), (order, i)
            assert same(eager.result(), eager_ref)
            assert same(layers[i].replayed(), ref[i]), (order, i)
    ctx.check_device()
    for lay in layers:
        del lay.graph
    torch.cuda.synchronize()


def test_table_rewritten_between_calls(E, oracle):
    """The same table buffer filled with other records (at lower and higher addresses) between two calls, and between two replays of a graph."""
    ctx = E.Context(flags=E.HB_FLAG_DECODE_TC_GU)
    lay = Layer(E, oracle, ctx, 4, 4, 2048, 512, seed=3)
    keep = lay.recs
    moved = [torch.empty_like(r) for r in keep]
    for a, b in zip(moved, reversed(keep)):
        a.copy_(b)
    first, second = E.rec_table(keep[:8]), E.rec_table(moved[:8])
    ref = [lay.result(ctx=E.Context(flags=E.HB_FLAG_DECODE_TC_GU), tab=t) for t in (first, second)]
    assert not same(*ref)
    lay.capture(True)
    for t, r in ((second, ref[1]), (first, ref[0]), (second, ref[1])):
        lay.tab.copy_(t)
        assert same(lay.result(), r)
        assert same(lay.replayed(), r)
    ctx.check_device()
    del lay.graph


@pytest.mark.parametrize("H,I,M,layer", [(2048, 512, 4, False), (512, 768, 8, False), (2048, 512, 70, True), (512, 768, 70, True)])
def test_records_at_any_16_byte_address(E, oracle, H, I, M, layer):
    """Records 16 bytes apart modulo everything (the alignment that record assembly asks for): the bits of the same records at 4096-byte
    addresses, through both kernels that read records by TMA."""
    flags = E.HB_FLAG_PREFILL_A16 if layer else E.HB_FLAG_DECODE_TC_GU
    lay = Layer(E, oracle, E.Context(flags=flags), M, 4, H, I, seed=H + I, layer=layer)
    n = lay.recs[0].numel()
    assert n % 4096 == 0

    def placed(shift):
        buf = torch.empty(9 * (n + 4096) + 4096, dtype=torch.uint8, device="cuda")
        at = -buf.data_ptr() % 4096
        out = []
        for i, r in enumerate(lay.recs):
            o = at + i * (n + 4096) + shift(i)
            buf[o:o + n] = r
            out.append(buf[o:o + n])
        return out

    ref = None
    for shift in (lambda i: 0, lambda i: 16, lambda i: 512 * (i % 3), lambda i: 16 * (7 * i % 61)):
        recs = placed(shift)
        got = lay.result(tab=E.rec_table(recs[:8]), shared=recs[8])
        lay.ctx.check_device()
        ref = got if ref is None else ref
        assert same(got, ref)


@pytest.mark.parametrize("M,layer", [(8, False), (70, True)])
def test_records_further_apart_than_a_map_reaches(E, oracle, M, layer):
    """Two allocations mapped 2^31 rows (256 GB of address space at 256 columns) apart: the boxes of the far ones are put together from small copies."""
    drv = pytest.importorskip("cuda.bindings.driver")

    def ok(r):
        assert r[0] == drv.CUresult.CUDA_SUCCESS, r[0]
        return r[1] if len(r) > 1 else None

    H = I = 256
    flags = E.HB_FLAG_PREFILL_A16 if layer else E.HB_FLAG_DECODE_TC_GU
    lay = Layer(E, oracle, E.Context(flags=flags), M, 4, H, I, seed=5, layer=layer)
    ref = lay.result()
    prop = drv.CUmemAllocationProp()
    prop.type = drv.CUmemAllocationType.CU_MEM_ALLOCATION_TYPE_PINNED
    prop.location.type = drv.CUmemLocationType.CU_MEM_LOCATION_TYPE_DEVICE
    prop.location.id = torch.cuda.current_device()
    chunk = ok(drv.cuMemGetAllocationGranularity(prop, drv.CUmemAllocationGranularity_flags.CU_MEM_ALLOC_GRANULARITY_MINIMUM))
    n = lay.recs[0].numel()
    chunk = max(chunk, -(-5 * n // chunk) * chunk)
    span = (H // 2) << 31
    acc = drv.CUmemAccessDesc()
    acc.location.type, acc.location.id = prop.location.type, prop.location.id
    acc.flags = drv.CUmemAccess_flags.CU_MEM_ACCESS_FLAGS_PROT_READWRITE
    va = int(ok(drv.cuMemAddressReserve(span + chunk, 0, 0, 0)))
    handles = [ok(drv.cuMemCreate(chunk, prop, 0)) for _ in range(2)]
    try:
        for h, base in zip(handles, (va, va + span)):
            ok(drv.cuMemMap(base, chunk, 0, h, 0))
            ok(drv.cuMemSetAccess(base, chunk, [acc], 1))
        addr = [(va if i % 2 == 0 else va + span) + (i // 2) * n for i in range(9)]
        for a, r in zip(addr, lay.recs):
            ok(drv.cuMemcpyDtoD(a, r.data_ptr(), n))
        torch.cuda.synchronize()
        for order in (addr, addr[1:8] + addr[:1] + addr[8:]):            # the shared expert near, then every record somewhere else
            tab = torch.tensor(order[:8], dtype=torch.int64, device="cuda")
            got = lay.result(tab=tab, shared=order[8])
            lay.ctx.check_device()
            if order is addr:
                assert same(got, ref)
            else:
                perm = E.rec_table(lay.recs[1:8] + lay.recs[:1])
                assert same(got, lay.result(tab=perm))
    finally:
        torch.cuda.synchronize()
        for h, base in zip(handles, (va, va + span)):
            drv.cuMemUnmap(base, chunk)
            drv.cuMemRelease(h)
        drv.cuMemAddressFree(va, span + chunk)
