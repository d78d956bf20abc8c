"""The work a user of this library has it do, as cases that can be timed and checked: decode steps over MoE layers, whole layers at
serving batches, prefill of token chunks with NVFP4 and with bf16 activations, the dense decode FFN in its three weight formats,
the dense prefill GEMM, the weight quantiser and the assembly of expert records.

Shapes are the repository's own configurations: "qwen" (hidden 2048, 512 experts top-10 + shared, intermediate 512, softmax router),
"glm" (hidden 4096, 160 experts top-8 + shared, intermediate 1536, sigmoid router with a skewed bias), "deepseek" (hidden 7168, 256
experts top-8, intermediate 2048) and the dense 5120 x 17408 FFN.  Weights are N(0, 0.02) quantised to the case's format, activations
bf16 N(0, 1), router logits N(0, 1).
"""
import math

import torch

import eke_hive_b200 as E

MODELS = {
    "qwen": dict(H=2048, I=512, E=512, K=10, router="softmax"),
    "glm": dict(H=4096, I=1536, E=160, K=8, router="sigmoid"),
    "deepseek": dict(H=7168, I=2048, E=256, K=8, router="softmax"),
}
GLM_SCALE = 2.5        # routed scaling factor of the sigmoid router
FMT = {"nvfp4": 0, "lb3": 1, "lb2": 2}
LB_BITS = {"lb3": 3, "lb2": 2}


def listed():
    return [
        # one sequence being generated: the latency of a step, replayed from the CUDA graph a decode loop keeps
        dict(name="decode_qwen_b1", kind="decode", model="qwen", rows=1, layers=6, graph=True),
        # a small serving batch, the size this library's benchmark quotes
        dict(name="decode_qwen_b16", kind="decode", model="qwen", rows=16, layers=6, graph=True),
        # big experts with hot ones among them, layers called one by one as an engine without graphs does
        dict(name="decode_glm_b8", kind="decode", model="glm", rows=8, layers=4, graph=False),
        # a full continuous-batching step of an odd number of sequences through the any-size layer call
        dict(name="layer_qwen_b45", kind="layer", model="qwen", rows=45, layers=4, graph=False),
        # one 8192-token prompt chunk with NVFP4 activations: the largest call
        dict(name="prefill_a4_deepseek_8192", kind="prefill_a4", model="deepseek", rows=8192),
        # a prompt of an odd length through a layer that keeps bf16 activations
        dict(name="prefill_a16_qwen_1999", kind="prefill_a16", model="qwen", rows=1999),
        # the dense FFN of a decode step: one sequence, a few sequences, in each weight format
        dict(name="dense_nvfp4_m1", kind="dense", fmt="nvfp4", rows=1, hidden=5120, ffn=17408, layers=3),
        dict(name="dense_lb3_m8", kind="dense", fmt="lb3", rows=8, hidden=5120, ffn=17408, layers=3),
        dict(name="dense_lb2_m3", kind="dense", fmt="lb2", rows=3, hidden=5120, ffn=17408, layers=3),
        # the dense FFN's gate matrix over a prompt chunk: activations quantised, then the FP4 GEMM
        dict(name="gemm_a4_4096", kind="gemm_a4", rows=4096, N=17408, K=5120),
        # a checkpoint being loaded: fp32 weights to NVFP4, and a layer's experts put together from their tensors
        dict(name="quantize_17408x5120", kind="quantize", N=17408, K=5120),
        dict(name="records_qwen_256", kind="records", model="qwen", n=256),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "decode", "layer", "prefill_a4", "prefill_a16", "dense", "dense", "dense", "gemm_a4", "quantize", "records"])
    if kind == "decode":
        return dict(kind=kind, model=rng.choice(["qwen", "qwen", "glm"]), rows=_log(rng, 1, 32), layers=rng.randint(3, 4), graph=rng.random() < 0.5)
    if kind == "layer":
        return dict(kind=kind, model=rng.choice(["qwen", "glm"]), rows=rng.randint(17, 64), layers=rng.randint(2, 4), graph=False)
    if kind == "prefill_a4":
        return dict(kind=kind, model=rng.choice(["qwen", "glm", "deepseek"]), rows=_log(rng, 200, 8000))
    if kind == "prefill_a16":
        return dict(kind=kind, model=rng.choice(["qwen", "glm"]), rows=_log(rng, 100, 4000))
    if kind == "dense":
        hidden, ffn = rng.choice([(5120, 17408), (5120, 13824), (4096, 12288), (2048, 6144)])
        return dict(kind=kind, fmt=rng.choice(["nvfp4", "lb3", "lb2"]), rows=rng.randint(1, 16), hidden=hidden, ffn=ffn, layers=rng.randint(2, 3))
    if kind == "gemm_a4":
        n, k = rng.choice([(17408, 5120), (5120, 17408), (8192, 8192), (6144, 2048)])
        return dict(kind=kind, rows=_log(rng, 300, 4000), N=n, K=k)
    if kind == "quantize":
        return dict(kind=kind, N=_log(rng, 1000, 17000), K=16 * rng.randint(100, 320))
    return dict(kind=kind, model=rng.choice(["qwen", "glm"]), n=_log(rng, 16, 200))


# ---------------------------------------------------------------------------------------------------- plain formats
_E2M1 = [0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0]


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _randn(g, *shape, dtype=torch.bfloat16):
    return torch.randn(shape, generator=g, device="cuda", dtype=torch.float32).to(dtype)


def _e2m1_codes(v):
    """Nearest e2m1 code of each value, ties to the even code."""
    edge = torch.tensor([0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5.0], device=v.device, dtype=v.dtype)
    a = v.abs()
    up, down = torch.bucketize(a, edge, right=True), torch.bucketize(a, edge, right=False)
    c = torch.where(up != down, torch.where(up % 2 == 0, up, down), up)
    return (c + 8 * torch.signbit(v)).to(torch.uint8)


def _pack4(c):
    return c[..., 0::2] | (c[..., 1::2] << 4)


def _quant_fp4(w, g):
    """w [..., K] with one scale g: (codes u8 [..., K / 2], e4m3 scales u8 [..., K / 16])."""
    b = w.reshape(*w.shape[:-1], -1, 16)
    s = ((b.abs().amax(-1) / 6.0) / g).clamp(max=448.0).to(torch.float8_e4m3fn)
    sf = s.to(w.dtype).unsqueeze(-1) * g
    c = _e2m1_codes(torch.where(sf > 0, b / torch.where(sf > 0, sf, torch.ones_like(sf)), torch.zeros_like(b)))
    return _pack4(c.reshape(w.shape)), s.view(torch.uint8)


def _nvfp4_matrix(g, N, K):
    w = torch.randn((N, K), generator=g, device="cuda") * 0.02
    gl = float(w.abs().max()) / (448.0 * 6.0)
    return (*_quant_fp4(w, gl), gl)


def _dequant(codes, scales, gl):
    """float64 [N, K] of NVFP4 codes u8 [N, K / 2] and scales u8 [N, K / 16]."""
    lut = torch.tensor(_E2M1 + [-v for v in _E2M1], dtype=torch.float64, device=codes.device)
    pair = torch.stack((lut.repeat(16), lut.repeat_interleave(16)), -1)            # byte -> (low nibble, high nibble)
    w = pair[codes.long()].reshape(codes.shape[0], -1, 16)
    return (w * (scales.view(torch.float8_e4m3fn).double() * gl).unsqueeze(-1)).reshape(codes.shape[0], -1)


def _lb_matrix(g, bits, N, K):
    """A group-64 low-bit matrix of N(0, 0.02) weights: (codes u8, scales f16 [N, K / 64], zero-points f16)."""
    w = (torch.randn((N, K), generator=g, device="cuda") * 0.02).reshape(N, K // 64, 64)
    lo, hi = w.amin(-1), w.amax(-1)
    s = ((hi - lo) / (2 ** bits - 1)).half()
    zp = (-lo / s.float()).half()
    q = (w / s.float().unsqueeze(-1) + zp.float().unsqueeze(-1)).round().clamp(0, 2 ** bits - 1).to(torch.uint8).reshape(N, K)
    l2 = q & 3
    low = l2[:, 0::4] | (l2[:, 1::4] << 2) | (l2[:, 2::4] << 4) | (l2[:, 3::4] << 6)
    if bits == 2:
        return low.contiguous().reshape(-1), s, zp
    h = (q >> 2).reshape(N, K // 8, 8)
    high = sum(h[:, :, j] << j for j in range(8)).to(torch.uint8)
    return torch.cat((low.reshape(-1), high.reshape(-1))), s, zp


def _lb_dequant(W, bits, N, K):
    q, s, zp = W
    low = q[:N * K // 4].reshape(N, K // 4, 1)
    v = ((low >> torch.tensor([0, 2, 4, 6], device=q.device, dtype=torch.uint8)) & 3).reshape(N, K)
    if bits == 3:
        high = q[N * K // 4:].reshape(N, K // 8, 1)
        v = v + 4 * ((high >> torch.arange(8, device=q.device, dtype=torch.uint8)) & 1).reshape(N, K)
    v = v.double().reshape(N, K // 64, 64)
    return ((v - zp.double().unsqueeze(-1)) * s.double().unsqueeze(-1)).reshape(N, K)


def _a4_rows(x):
    """Rows in float64 as the activation quantiser leaves them: one fp32 scale per row, one e4m3 scale per 16 values, e2m1 codes."""
    f = x.float()
    amax = f.abs().amax(-1, keepdim=True)
    gx = torch.where(amax > 0, amax / torch.full_like(amax, 2688.0), torch.ones_like(amax))    # tensors: a division by a number would be a product
    inv = torch.ones_like(gx) / gx
    b = f.reshape(f.shape[0], -1, 16)
    m = b.abs().amax(-1)
    s = ((m / torch.full_like(m, 6.0)) * inv).clamp(max=448.0).to(torch.float8_e4m3fn)
    sf = s.float()
    fac = torch.where(sf > 0, inv / torch.where(sf > 0, sf, torch.ones_like(sf)), torch.zeros_like(sf))
    c = _e2m1_codes(b * fac.unsqueeze(-1))
    lut = torch.tensor(_E2M1 + [-v for v in _E2M1], dtype=torch.float64, device=x.device)
    return (lut[c.long()] * sf.double().unsqueeze(-1)).reshape(f.shape) * gx.double()


# ---------------------------------------------------------------------------------------------------- inputs
_CONTEXTS = {}


def _context(flags=0):
    if flags not in _CONTEXTS:
        _CONTEXTS[flags] = E.Context(flags=flags)
    return _CONTEXTS[flags]


def _experts(g, H, I, n):
    """n expert records u8 [n, total] in the library's layout: quantised N(0, 0.02) blocks drawn from a pool, their own scales with them."""
    lay = E.ExpertRecLayout(H, I)
    chunk, pool = 8192, 2048                                     # values per chunk; all three matrices hold whole chunks
    codes, scales, gl = _nvfp4_matrix(g, pool, chunk)
    recs = torch.zeros((n, lay.total), dtype=torch.uint8, device="cuda")
    nch = H * I // chunk
    step = max(1, (1 << 30) // (nch * chunk // 2))
    for a in range(0, n, step):
        b = min(n, a + step)
        for w_off, s_off in ((lay.w1, lay.s1), (lay.w3, lay.s3), (lay.w2, lay.s2)):
            at = torch.randint(0, pool, ((b - a) * nch,), generator=g, device="cuda")
            recs[a:b, w_off:w_off + H * I // 2] = codes[at].reshape(b - a, -1)
            recs[a:b, s_off:s_off + H * I // 16] = scales[at].reshape(b - a, -1)
    glob = gl * (0.8 + 0.4 * torch.rand((n, 3), generator=g, device="cuda"))
    recs[:, lay.g:lay.g + 12] = glob.view(torch.uint8)
    return recs


def _moe_inputs(case, seed):
    m, g = MODELS[case["model"]], _gen(seed)
    L, B = case.get("layers", 1), case["rows"]
    n = m["E"] + 1                                                # the shared expert is the last record of a layer
    recs = _experts(g, m["H"], m["I"], L * n)
    softmax = m["router"] == "softmax"
    logits = torch.randn((L, B, n if softmax else m["E"]), generator=g, device="cuda")     # softmax: the last column gates the shared expert
    bias = None
    if not softmax:
        z = 1.0 / torch.arange(1, m["E"] + 1, device="cuda", dtype=torch.float64) ** 1.1
        bias = torch.log(z / z.sum()).float()[torch.randperm(m["E"], generator=g, device="cuda")].contiguous()
    x = _randn(g, L, B, m["H"])
    ptr = recs.data_ptr() + recs.stride(0) * torch.arange(L * n, dtype=torch.int64).reshape(L, n)
    tab = ptr[:, :m["E"]].contiguous().cuda()
    return dict(m=m, L=L, B=B, recs=recs, logits=logits, bias=bias, x=x, tab=tab, shared=[int(p) for p in ptr[:, m["E"]]], softmax=softmax)


def _layer_call(s, li, call, ctx):
    m = s["m"]
    call(s["logits"][li], s["x"][li], s["tab"], li, m["E"], m["K"], m["H"], m["I"], shared_rec=s["shared"][li],
         gate_col=m["E"] if s["softmax"] else -1, bias=s["bias"], sigmoid_scale=0.0 if s["softmax"] else GLM_SCALE,
         ids=s["ids"][li], w=s["w"][li], out=s["out"][li], ws=s["ws"], ctx=ctx)


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("decode", "layer", "prefill_a16"):
        s = _moe_inputs(case, seed)
        m, L, B = s["m"], s["L"], s["B"]
        s["ids"] = torch.zeros((L, B, m["K"]), dtype=torch.int32, device="cuda")
        s["w"] = torch.zeros((L, B, m["K"]), device="cuda")
        s["out"] = torch.zeros((L, B, m["H"]), dtype=torch.bfloat16, device="cuda")
        nws = E.moe_decode_ws_bytes(B * (m["K"] + 1), m["H"], m["I"]) if kind == "decode" else E.moe_layer_ws_bytes(B, m["K"], m["E"], m["H"], m["I"])
        s["ws"] = torch.empty(nws, dtype=torch.uint8, device="cuda")
        s["call"] = E.moe_layer_decode if kind == "decode" else E.moe_layer
        s["ctx"] = _context(E.HB_FLAG_PREFILL_A16 if kind == "prefill_a16" else 0)
        if case.get("graph"):
            side = torch.cuda.Stream()
            side.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(side):
                for li in range(L):
                    _layer_call(s, li, s["call"], s["ctx"])
            torch.cuda.current_stream().wait_stream(side)
            s["graph"] = torch.cuda.CUDAGraph()
            with torch.cuda.graph(s["graph"]):
                for li in range(L):
                    _layer_call(s, li, s["call"], s["ctx"])
    elif kind == "prefill_a4":
        s = _moe_inputs(case, seed)
        m, B = s["m"], s["B"]
        s["w"], ids = torch.topk(torch.softmax(s["logits"][0, :, :m["E"]], -1), m["K"])
        s["ids"] = ids.int().contiguous()
        s["out"] = torch.zeros((B, m["H"]), device="cuda")
        s["ws"] = torch.empty(E.moe_prefill_ws_bytes(B, m["K"], m["E"], m["H"], m["I"]), dtype=torch.uint8, device="cuda")
        s["ctx"] = _context()
    elif kind == "dense":
        g, s = _gen(seed), dict(layers=[], ctx=_context())
        fmt, M, H, F = FMT[case["fmt"]], case["rows"], case["hidden"], case["ffn"]
        for _ in range(case["layers"]):
            mats = [_dense_matrix(g, case["fmt"], N, K) for N, K in ((F, H), (F, H), (H, F))]
            gate, up, down = (E.GMat(fmt, N, K, *(W[:2] if fmt == 0 else W), **({"g": W[2]} if fmt == 0 else {}))
                              for W, (N, K) in zip(mats, ((F, H), (F, H), (H, F))))
            s["layers"].append(dict(mats=mats, gate=gate, up=up, down=down, x=_randn(g, M, H), act=torch.zeros((M, F), dtype=torch.bfloat16, device="cuda"),
                                    y=torch.zeros((M, H), device="cuda")))
        s["ws"] = torch.empty(max(E.dense_gemv_ws_bytes(fmt, F, H, 2), E.dense_gemv_ws_bytes(fmt, H, F, 1)), dtype=torch.uint8, device="cuda")
    elif kind == "gemm_a4":
        g = _gen(seed)
        W = _nvfp4_matrix(g, case["N"], case["K"])
        s = dict(W=W, mat=E.GMat(0, case["N"], case["K"], W[0], W[1], g=W[2]), x=_randn(g, case["rows"], case["K"]),
                 y=torch.zeros((case["rows"], case["N"]), device="cuda"), ctx=_context())
    elif kind == "quantize":
        N, K = case["N"], case["K"]
        s = dict(weight=torch.randn((N, K), generator=_gen(seed), device="cuda") * 0.02, q=torch.zeros((N, K // 2), dtype=torch.uint8, device="cuda"),
                 s=torch.zeros((N, K // 16), dtype=torch.uint8, device="cuda"), g=torch.zeros(1, device="cuda"), ctx=_context())
    else:
        s = _record_sources(case, seed)
        m, n = s["m"], case["n"]
        s["out"] = torch.zeros((n, E.ExpertRecLayout(m["H"], m["I"]).total), dtype=torch.uint8, device="cuda")
        s["jobs"] = E.record_jobs(s["experts"], s["out"])
        s["status"] = torch.full((n, 3, 2), -1, dtype=torch.int32, device="cuda")
        s["ws"] = torch.empty(max(E.record_pack_ws_bytes(m["H"], m["I"], n), 256), dtype=torch.uint8, device="cuda")
        s["n"], s["ctx"] = n, _context()
    s["kind"] = kind
    return s


def _dense_matrix(g, fmt, N, K):
    return _nvfp4_matrix(g, N, K) if fmt == "nvfp4" else _lb_matrix(g, LB_BITS[fmt], N, K)


def _csf(g, R, C):
    """Compressed block scales of R x C codes: 16 row bases and 4-bit deltas per 16 rows, 2 % of the entries outside the deltas' reach."""
    base = torch.randint(38, 44, (R // 16, 16), generator=g, device="cuda", dtype=torch.int32).to(torch.uint8)
    delta = torch.randint(0, 16, (R // 16, 16 * C), generator=g, device="cuda", dtype=torch.int32).to(torch.uint8)
    far = torch.rand((R // 16, 16 * C), generator=g, device="cuda") < 0.02
    delta[far] = 0
    at = far.reshape(-1).nonzero().reshape(-1)
    code = torch.randint(64, 0x7F, (at.numel(),), generator=g, device="cuda")
    word = (code << 24) | at
    return torch.cat((base, _pack4(delta)), 1).contiguous(), word.to(torch.int32)


def _record_sources(case, seed):
    m, g = MODELS[case["model"]], _gen(seed)
    shapes = ((m["I"], m["H"]), (m["I"], m["H"]), (m["H"], m["I"]))
    fixed = [[_csf(g, R, K // 16) for R, K in shapes] for _ in range(8)]           # eight patterns, in memory of its own for each expert
    experts = []
    for i in range(case["n"]):
        experts.append([dict(weight=torch.randint(0, 256, (R, K // 2), generator=g, device="cuda", dtype=torch.uint8), csf_fixed=f.clone(), csf_exc=e.clone(),
                             **{"global": 1e-4 * (1 + j + i % 3)}) for j, ((R, K), (f, e)) in enumerate(zip(shapes, fixed[i % 8]))])
    return dict(m=m, experts=experts)


# ---------------------------------------------------------------------------------------------------- one pass
def run(s):
    kind = s["kind"]
    if kind in ("decode", "layer", "prefill_a16"):
        if "graph" in s:
            s["graph"].replay()
        else:
            for li in range(s["L"]):
                _layer_call(s, li, s["call"], s["ctx"])
        return dict(ids=s["ids"], w=s["w"], out=s["out"])
    if kind == "prefill_a4":
        m = s["m"]
        return E.fn_moe_prefill(s["tab"], 0, m["E"], s["ids"], s["w"], s["x"][0], m["H"], m["I"], out=s["out"], ws=s["ws"], ctx=s["ctx"])
    if kind == "dense":
        out = []
        for p in s["layers"]:
            E.dense_gemv_gu(p["gate"], p["up"], p["x"], act=p["act"], ws=s["ws"], ctx=s["ctx"])
            E.dense_gemv(p["down"], p["act"], y=p["y"], ws=s["ws"], ctx=s["ctx"])
            out.append(dict(act=p["act"], y=p["y"]))
        return out
    if kind == "gemm_a4":
        q, sc, g = E.a4_quant(s["x"], ctx=s["ctx"])
        return dict(q=q, s=sc, g=g, y=E.nvfp4_gemm_a4(s["mat"], q, sc, g, y=s["y"], ctx=s["ctx"]))
    if kind == "quantize":
        q, sc, g = E.nvfp4_quantize(s["weight"], q=s["q"], s=s["s"], g=s["g"], ctx=s["ctx"])
        return dict(q=q, s=sc, g=g)
    E.record_pack_batch(s["jobs"], s["n"], s["m"]["H"], s["m"]["I"], status=s["status"], ws=s["ws"], ctx=s["ctx"])
    return dict(recs=s["out"], status=s["status"])


# ---------------------------------------------------------------------------------------------------- what a pass needs
def _distinct(m, rows):
    """Experts that a call of so many rows touches, on average; for the skewed router those of a sample."""
    if m["router"] == "softmax":
        return m["E"] * (1.0 - (1.0 - m["K"] / m["E"]) ** rows)
    z = 1.0 / torch.arange(1, m["E"] + 1, dtype=torch.float64) ** 1.1
    lg = torch.randn((rows, m["E"]), generator=torch.Generator().manual_seed(0), dtype=torch.float64)
    return float(torch.unique(torch.topk(torch.sigmoid(lg) + torch.log(z / z.sum()), m["K"]).indices).numel())


def work(case):
    kind = case["kind"]
    if kind in ("decode", "layer", "prefill_a16", "prefill_a4"):
        m, L, B = MODELS[case["model"]], case.get("layers", 1), case["rows"]
        shared = 0 if kind == "prefill_a4" else 1
        rec = 3 * m["H"] * m["I"] * 9 / 16 + 12
        io = B * m["H"] * 4 + B * m["K"] * 8 + (B * m["E"] * 4 if shared else 0) + (B * m["H"] * 2 if kind == "prefill_a4" else 0)
        return {"bytes": L * ((_distinct(m, B) + shared) * rec + io), "flops": L * 6.0 * m["H"] * m["I"] * B * (m["K"] + shared)}
    if kind == "dense":
        H, F, M = case["hidden"], case["ffn"], case["rows"]
        per = {"nvfp4": 9 / 16, "lb3": 7 / 16, "lb2": 5 / 16}[case["fmt"]]
        return {"bytes": case["layers"] * (3 * H * F * per + M * (H * 2 + F * 4 + H * 4)), "flops": case["layers"] * 6.0 * H * F * M}
    if kind == "gemm_a4":
        M, N, K = case["rows"], case["N"], case["K"]
        return {"bytes": N * K * 9 / 16 + M * K * 2 + M * K * 9 / 16 + 4 * M + M * N * 4, "flops": 2.0 * M * N * K}
    if kind == "quantize":
        return {"bytes": case["N"] * case["K"] * (4 + 9 / 16), "flops": 0}
    m = MODELS[case["model"]]
    return {"bytes": case["n"] * m["H"] * m["I"] * 3 * (0.5 + 0.035 + 9 / 16), "flops": 0}


def tolerance(case):
    kind = case["kind"]
    if kind in ("quantize", "records"):
        return "exact"                                            # bytes, and one scale that is a division of an exact maximum
    if kind == "gemm_a4":
        return {"rel": 1e-5, "max": 1e-4, "differ": 0.0}          # exact products, fp32 sums
    if kind == "prefill_a4":
        return {"rel": 6e-3, "max": 0.5, "differ": 0.0}           # a sum that rounds the other way can move a value of y to the next FP4 code
    return {"rel": 4e-3, "max": 0.06, "differ": 0.0}              # bf16 between the passes and at the end


# ---------------------------------------------------------------------------------------------------- 64 bits
def _topk_first(v, k):
    """The k largest of each row, the smaller index first among equals."""
    return torch.sort(v, dim=-1, descending=True, stable=True).indices[:, :k]


def _silu_mul(g, u):
    return g / (1.0 + torch.exp(-g)) * u


def _expert64(rec, lay, H, I):
    gl = rec[lay.g:lay.g + 12].view(torch.float32).double()
    mats = []
    for j, (w, sc, n, k) in enumerate(((lay.w1, lay.s1, I, H), (lay.w3, lay.s3, I, H), (lay.w2, lay.s2, H, I))):
        mats.append(_dequant(rec[w:w + n * k // 2].reshape(n, k // 2), rec[sc:sc + n * k // 16].reshape(n, k // 16), gl[j]))
    return mats


def _routed64(s, li, ids, w, x, a4):
    m = s["m"]
    lay = E.ExpertRecLayout(m["H"], m["I"])
    out = torch.zeros((x.shape[0], m["H"]), dtype=torch.float64, device="cuda")
    for e in torch.unique(ids).tolist():
        rows, pick = (ids == e).nonzero(as_tuple=True)
        w1, w3, w2 = _expert64(s["recs"][li * (m["E"] + 1) + e], lay, m["H"], m["I"])
        y = _silu_mul(x[rows] @ w1.T, x[rows] @ w3.T)
        if a4:
            y = _a4_rows(y)
        out.index_add_(0, rows, (y @ w2.T) * w[rows, pick].double().unsqueeze(-1))
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind in ("decode", "layer", "prefill_a16"):
        s = _moe_inputs(case, seed)
        m, L, B = s["m"], s["L"], s["B"]
        res = dict(ids=[], w=[], out=[])
        for li in range(L):
            lg = s["logits"][li]
            if s["softmax"]:
                p = torch.softmax(lg[:, :m["E"]].bfloat16().double(), -1)
                ids = _topk_first(p, m["K"])
                w = p.gather(1, ids)
                w = w / w.sum(-1, keepdim=True)
                gate = torch.sigmoid(lg[:, m["E"]].bfloat16().double())
            else:
                p = torch.sigmoid(lg.double())
                ids = _topk_first(p + s["bias"].double(), m["K"])
                w = p.gather(1, ids)
                w = w / (w.sum(-1, keepdim=True) + 1e-20) * GLM_SCALE
                gate = torch.ones(B, dtype=torch.float64, device="cuda")
            x = s["x"][li].double()
            out = _routed64(s, li, ids, w, x, False)
            w1, w3, w2 = _expert64(s["recs"][li * (m["E"] + 1) + m["E"]], E.ExpertRecLayout(m["H"], m["I"]), m["H"], m["I"])
            out += (_silu_mul(x @ w1.T, x @ w3.T) @ w2.T) * gate.unsqueeze(-1)
            res["ids"].append(ids.int())
            res["w"].append(w)
            res["out"].append(out)
        return {k: torch.stack(v) for k, v in res.items()}
    if kind == "prefill_a4":
        s = _moe_inputs(case, seed)
        m = s["m"]
        w, ids = torch.topk(torch.softmax(s["logits"][0, :, :m["E"]], -1), m["K"])
        return _routed64(s, 0, ids, w, _a4_rows(s["x"][0]), True)
    if kind == "dense":
        g, res = _gen(seed), []
        M, H, F, fmt = case["rows"], case["hidden"], case["ffn"], case["fmt"]
        for _ in range(case["layers"]):
            mats = [_dense_matrix(g, fmt, N, K) for N, K in ((F, H), (F, H), (H, F))]
            x = _randn(g, M, H).double()
            deq = (lambda W, N, K: _dequant(*W)) if fmt == "nvfp4" else (lambda W, N, K: _lb_dequant(W, LB_BITS[fmt], N, K))
            act = _silu_mul(x @ deq(mats[0], F, H).T, x @ deq(mats[1], F, H).T)
            res.append(dict(act=act, y=act @ deq(mats[2], H, F).T))
        return res
    if kind == "gemm_a4":
        g = _gen(seed)
        W = _nvfp4_matrix(g, case["N"], case["K"])
        x = _randn(g, case["rows"], case["K"])
        return dict(q=None, s=None, g=(x.double().abs().amax(-1) / 2688.0), y=_a4_rows(x) @ _dequant(*W).T)
    if kind == "quantize":
        w = torch.randn((case["N"], case["K"]), generator=_gen(seed), device="cuda") * 0.02
        return dict(q=None, s=None, g=(w.double().abs().max() / 2688.0).reshape(1))
    return None
