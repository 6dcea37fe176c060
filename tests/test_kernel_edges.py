"""Sizes at which the kernels of the layer change form or run out of tile: token counts around
32 / 64 / 128, lists that are empty, single or everything, widths outside the multiples the
wide forms take.  Against the CPU oracle, with the tolerances of the parity tests."""
import numpy as np
import pytest
import torch

from helpers import C, O, TOL, WINDOW

pytestmark = pytest.mark.gpu


def _gen(seed):
    return torch.Generator().manual_seed(seed)


def _layer(N, d, H, E, R, dtype, seed, act="relu", glu=False, mask_p=None):
    c = C.LayerCase("edge", 1, N, d, H, E, R=R, dtype=dtype, act=act, glu=glu, seed=seed,
                    zero_last_bias=glu)
    return c, C.make_tensors(c)


def _dev(t):
    return None if t is None else t.cuda().contiguous()


def _lists(wsp, E):
    off = wsp.offsets.cpu().numpy()
    return off, wsp.token_idx[: int(off[E])].cpu().numpy()


def _mask(kind, N, E, g):
    if kind == "one_expert":                  # every token to one expert, the others empty
        m = torch.zeros(N, E, dtype=torch.bool)
        m[:, E // 2] = True
    elif kind == "all":
        m = torch.ones(N, E, dtype=torch.bool)
    elif kind == "first_token":               # lists of one row or none
        m = torch.zeros(N, E, dtype=torch.bool)
        m[0] = True
    else:
        m = torch.rand(N, E, generator=g) < 0.3
    return m


EXPERTS = [  # N, d, H, E, activation, gated
    (1, 64, 16, 1, "relu", False), (31, 192, 48, 5, "gelu", False), (32, 128, 128, 7, "relu", False),
    (33, 320, 32, 3, "tanh", False), (64, 768, 128, 4, "relu", False), (65, 128, 80, 6, "relu", False),
    (127, 256, 128, 2, "leaky_relu", False), (129, 768, 32, 128, "relu", False),
    (1, 128, 128, 4, "gelu", True), (32, 256, 128, 9, "gelu", True), (65, 192, 64, 3, "gelu", True),
    (300, 256, 128, 5, "gelu", True),
]


@pytest.mark.parametrize("kind", ["random", "one_expert", "all", "first_token"])
@pytest.mark.parametrize("N,d,H,E,act,glu", EXPERTS)
def test_tensor_core_experts(N, d, H, E, act, glu, kind):
    from d2dmoe_b200 import ops
    c, t = _layer(N, d, H, E, 128, "bf16", N + d, act, glu)
    m = _mask(kind, N, E, _gen(N))
    wsp = ops.Workspace.allocate(N, E, "cuda")
    wsp.mask_bits[:N].copy_(torch.from_numpy(O.pack_mask(m).view(np.int32)).cuda())
    ops.compact(wsp, N, E)
    w1, b1, w2, wu = (_dev(t.get(k)) for k in ("w1", "b1", "w2", "w_up"))
    if glu:
        b1 = None
    packed = ops.prepack_experts(w1, b1, w2, wu)
    assert packed is not None
    x2d = _dev(t["x"].reshape(N, d))
    out = torch.full((N, d), float("nan"), dtype=torch.bfloat16, device="cuda")
    norms = torch.full((E, N), float("nan"), dtype=torch.bfloat16, device="cuda")
    ex = O.experts_ffn_exact(t["x"].reshape(N, d), m, t["w1"], None if glu else t["b1"], t["w2"], act,
                             t.get("w_up") if glu else None)
    for kw in ({}, dict(norms=norms, norm_layer="output"), dict(norms=norms, norm_layer="intermediate")):
        ops.experts_ffn(x2d, wsp, w1, b1, w2, act, out, w_up=wu, packed=packed, **kw)
        wsp.check_status()
        o = out.cpu().float()
        assert torch.isfinite(o).all()
        # k bf16 adds per element, each rounding at the running magnitude
        assert O.rel_err(o, ex) <= TOL["bf16"] * max(1.0, m.sum(1).max().item() ** 0.5 / 2)
        if kw:
            ref = O.expert_activation_norms(t["x"].reshape(N, d), t["w1"], None if glu else t["b1"],
                                            t["w2"], act, t.get("w_up") if glu else None,
                                            layer=kw["norm_layer"], ord=2).float()
            assert O.rel_err(norms.cpu().float(), torch.where(m.t(), ref, 0.0)) <= TOL["bf16"]


SHORT = [  # N, d, H, E, activation, gated: around 32 rows of a list, every cluster form, several rounds
    (1, 128, 32, 3, "relu", False), (31, 256, 64, 24, "gelu", False), (33, 768, 96, 6, "tanh", False),
    (64, 384, 128, 5, "leaky_relu", False), (65, 2048, 128, 20, "relu", False),
    (32, 384, 96, 3, "gelu_tanh", True), (33, 640, 32, 9, "gelu", True), (40, 256, 64, 5, "relu", True),
    (257, 2048, 128, 128, "gelu", True), (512, 2048, 128, 128, "gelu", True),
    # CTAs without output columns (d < 512), more items than clusters
    (512, 128, 32, 10, "relu", False), (511, 256, 128, 10, "gelu", True), (500, 384, 64, 9, "relu", False),
]


@pytest.mark.parametrize("kind", ["one_expert", "first_token", "few", "random", "all"])
@pytest.mark.parametrize("N,d,H,E,act,glu", SHORT)
def test_short_call_experts(N, d, H, E, act, glu, kind):
    from d2dmoe_b200 import ops
    c, t = _layer(N, d, H, E, 128, "bf16", N + d, act, glu)
    g = _gen(N)
    m = torch.rand(N, E, generator=g) < 2.0 / E if kind == "few" else _mask(kind, N, E, g)
    if kind in ("random", "all") and E > 64:  # lists of up to about 90 rows, the oracle in bounds
        m &= torch.rand(1, E, generator=g) < 0.2
    wsp = ops.Workspace.allocate(N, E, "cuda")
    wsp.mask_bits[:N].copy_(torch.from_numpy(O.pack_mask(m).view(np.int32)).cuda())
    ops.compact(wsp, N, E)
    w1, b1, w2, wu = (_dev(t.get(k)) for k in ("w1", "b1", "w2", "w_up"))
    if glu:
        b1 = None
    packed = ops.prepack_experts(w1, b1, w2, wu)
    x2d = _dev(t["x"].reshape(N, d))
    out = torch.full((N, d), float("nan"), dtype=torch.bfloat16, device="cuda")
    ex = O.experts_ffn_exact(t["x"].reshape(N, d), m, t["w1"], None if glu else t["b1"], t["w2"], act,
                             t.get("w_up") if glu else None)
    ops.experts_ffn(x2d, wsp, w1, b1, w2, act, out, w_up=wu, packed=packed)
    wsp.check_status()
    o = out.cpu().float()
    assert torch.isfinite(o).all()
    # k bf16 adds per element, each rounding at the running magnitude
    assert O.rel_err(o, ex) <= TOL["bf16"] * max(1.0, m.sum(1).max().item() ** 0.5 / 2)


@pytest.mark.parametrize("E", [8, 24, 128])
@pytest.mark.parametrize("N,d", [(n, 2048) for n in (1, 31, 33, 128, 129, 700, 1921, 2048, 2049)] +
                         [(1920, 1024), (1921, 1024)])
def test_large_router(N, d, E):
    """Router d -> 256 -> E: split over clusters for short calls (up to 16 tiles, d < 2048 up to 15)."""
    from d2dmoe_b200 import ops
    R, tau = 256, 0.1
    c, t = _layer(N, d, 128, E, R, "bf16", N + E)
    x2d, wa, wb = _dev(t["x"].reshape(N, d)), _dev(t["wa"]), _dev(t["wb"])
    lb = _dev(t["last_bias"].reshape(-1))
    packed = ops.prepack_router(wa, wb)
    wsp = ops.Workspace.allocate(N, E, "cuda")
    sc = torch.empty(N, E, dtype=torch.bfloat16, device="cuda")
    out = torch.full((N, d), float("nan"), dtype=torch.bfloat16, device="cuda")
    for residual in (False, True):
        ops.router_mask(x2d, wa, wb, tau, wsp, packed=packed, scores_out=sc, last_bias=lb,
                        add_residual=residual, out_init=out)
        wsp.check_status()
        ref = O.router_scores(t["x"].reshape(N, d), t["wa"], t["wb"])
        assert O.rel_err(sc.cpu(), ref) <= 2.0 ** -7
        m = O.unpack_mask(wsp.mask_bits[:N].cpu().numpy().view(np.uint32), E)
        assert torch.equal(m, O.dynk_max_mask(sc.cpu(), tau))
        want = lb.float().expand(N, d) + (x2d.float() if residual else 0.0)
        assert torch.equal(out, want.to(torch.bfloat16))
    # the whole layer: lists of that mask, every row of the output written
    w1, b1, w2 = _dev(t["w1"]), _dev(t["b1"]), _dev(t["w2"])
    out.fill_(float("nan"))
    rt = torch.empty(N, E, dtype=torch.bfloat16, device="cuda")
    ops.moe_forward(x2d, wa, wb, tau, w1, b1, w2, "relu", out, wsp, last_bias=lb,
                    router_packed=packed, experts_packed=ops.prepack_experts(w1, b1, w2),
                    routing_out=rt)
    wsp.check_status()
    assert torch.equal(rt.cpu() > 0, m)
    off, idx = _lists(wsp, E)
    roff, ridx = O.expert_token_lists(m)
    assert np.array_equal(off, np.asarray(roff)) and np.array_equal(idx, np.asarray(ridx))
    ex = O.experts_ffn_exact(t["x"].reshape(N, d), m, t["w1"], t["b1"], t["w2"])
    assert O.rel_err(out.cpu().float(), ex + t["last_bias"].double()) <= TOL["bf16"]


@pytest.mark.parametrize("N,d,H,E,R", [(1, 4, 4, 1, 4), (31, 68, 36, 5, 36), (33, 260, 100, 33, 100),
                                       (64, 768, 128, 24, 128), (95, 132, 32, 256, 160),
                                       (257, 64, 64, 40, 64), (191, 256, 32, 1, 64), (192, 320, 96, 1, 128),
                                       (225, 4, 4, 1, 4), (417, 132, 100, 2, 36), (385, 516, 44, 2, 64)])
def test_fp32_layer(N, d, H, E, R):
    from d2dmoe_b200 import ops
    c, t = _layer(N, d, H, E, R, "fp32", N + d, act="gelu")
    x2d, wa, wb = _dev(t["x"].reshape(N, d)), _dev(t["wa"]), _dev(t["wb"])
    w1, b1, w2, lb = (_dev(t[k]) for k in ("w1", "b1", "w2", "last_bias"))
    wsp = ops.Workspace.allocate(N, E, "cuda")
    sc = torch.empty(N, E, device="cuda")
    ops.router_mask(x2d, wa, wb, 0.3, wsp, scores_out=sc)
    ref = O.router_scores(t["x"].reshape(N, d), t["wa"], t["wb"])
    assert O.rel_err(sc.cpu(), ref) <= TOL["fp32"]
    m = O.unpack_mask(wsp.mask_bits[:N].cpu().numpy().view(np.uint32), E)
    assert torch.equal(m, O.dynk_max_mask(sc.cpu(), 0.3))
    assert ((m != O.dynk_max_mask(ref, 0.3)) & ~O.near_threshold(ref, 0.3, WINDOW["fp32"])).sum() == 0
    for residual in (False, True):
        out = torch.full((N, d), float("nan"), device="cuda")
        rt = torch.empty(N, E, device="cuda")
        ops.moe_forward(x2d, wa, wb, 0.3, w1, b1, w2, "gelu", out, wsp, last_bias=lb.reshape(-1),
                        add_residual=residual, routing_out=rt)
        wsp.check_status()
        assert torch.equal(rt.cpu() > 0, m)
        ex = O.experts_ffn_exact(t["x"].reshape(N, d), m, t["w1"], t["b1"], t["w2"], "gelu")
        ex = ex + t["last_bias"].double() + (t["x"].reshape(N, d).double() if residual else 0.0)
        assert O.rel_err(out.cpu(), ex) <= TOL["fp32"]


@pytest.mark.parametrize("dtype,E", [("bf16", 8), ("bf16", 24), ("bf16", 64), ("bf16", 72),
                                     ("fp32", 4), ("fp32", 24), ("fp32", 32), ("fp32", 36)])
@pytest.mark.parametrize("N", [1, 127, 129, 300])
def test_every_mode_is_one_call(N, dtype, E):
    """topk / dynk / all through the one-call layer: the same mask as the rule kernel alone (which
    the upstream fixtures pin) on the layer's own scores, its lists, every output row."""
    import d2dmoe_b200 as D
    from d2dmoe_b200 import ops
    c, t = _layer(N, 128, 32, E, 64, dtype, N + E)
    moe = D.MoeficationMoE("m", c.d, E, True, c.H, torch.nn.ReLU)
    moe.router = D.MoeficationRouter(c.d, E, width=64, depth=2, bias=False, activation="relu",
                                     output_activation="abs")
    moe = moe.to(c.torch_dtype)
    moe.load_state_dict({"experts.w1": t["w1"], "experts.b1": t["b1"], "experts.w2": t["w2"],
                         "last_bias": t["last_bias"], "router.layers.0.weight": t["wa"],
                         "router.layers.2.weight": t["wb"]})
    moe = moe.cuda().eval()
    x, x2d = t["x"].cuda(), t["x"].reshape(N, c.d)
    wsp = ops.Workspace.allocate(N, E, "cuda")
    sc = torch.empty(N, E, dtype=c.torch_dtype, device="cuda")
    ops.router_mask(x.reshape(N, c.d), _dev(t["wa"]), _dev(t["wb"]), 0.5, wsp, scores_out=sc,
                    packed=moe.router.packed())
    for mode, k, tau in (("topk", 1, None), ("topk", min(3, E), None), ("topk", E, None),
                         ("dynk", None, 0.0), ("dynk", None, 0.45), ("dynk", None, 2.0),
                         ("all", None, None)):
        moe.forward_mode, moe.k, moe.tau = mode, k, tau
        out, gd = moe(x)
        got = gd["m"][0].reshape(N, E).cpu() > 0
        if mode == "all":
            want = torch.ones(N, E, dtype=torch.bool)
        else:
            ops.mask_rule_from_scores(sc, mode, wsp, k=k, tau=tau)
            want = O.unpack_mask(wsp.mask_bits[:N].cpu().numpy().view(np.uint32), E)
        assert torch.equal(got, want), (mode, k, tau)
        w = moe.last_workspace(N, x.device)
        w.check_status()
        off, idx = _lists(w, E)
        roff, ridx = O.expert_token_lists(want)
        assert np.array_equal(off, np.asarray(roff)) and np.array_equal(idx, np.asarray(ridx))
        ex = O.experts_ffn_exact(x2d, want, t["w1"], t["b1"], t["w2"]) + t["last_bias"].double()
        # bf16: k adds, each rounding at the running magnitude
        slack = max(1.0, want.sum(1).max().item() ** 0.5 / 2) if dtype == "bf16" else 1.0
        assert O.rel_err(out.reshape(N, c.d).cpu().float(), ex) <= TOL[dtype] * slack


@pytest.mark.parametrize("N,E", [(33, 1), (129, 16), (1025, 17), (1025, 31), (1200, 32), (1100, 33)])
def test_router_ranks_its_scores(N, E):
    """Up to 32 experts the router applies topk / dynk itself; lists inside and outside the cluster."""
    test_every_mode_is_one_call(N, "bf16", E)


@pytest.mark.parametrize("N,E", [(8192, 24), (8193, 24), (4096, 33), (4097, 33), (255, 256), (2100, 128)])
def test_compaction_with_and_without_table(N, E):
    from d2dmoe_b200 import ops
    m = torch.rand(N, E, generator=_gen(E)) < 0.1
    wsp = ops.Workspace.allocate(N, E, "cuda")
    wsp.mask_bits[:N].copy_(torch.from_numpy(O.pack_mask(m).view(np.int32)).cuda())
    ops.compact(wsp, N, E)
    wsp.check_status()
    off, idx = _lists(wsp, E)
    roff, ridx = O.expert_token_lists(m)
    assert np.array_equal(off, np.asarray(roff)) and np.array_equal(idx, np.asarray(ridx))


@pytest.mark.parametrize("E", [1, 24, 33, 128])
@pytest.mark.parametrize("N", [1, 128, 129, 1000, 1024, 1025])
def test_short_calls_write_their_lists(N, E):
    """Up to 1024 tokens the router kernel leaves the lists itself (one cluster), beyond that the
    scatter kernel does: lists, offsets and routing tensor of the mask either way."""
    from d2dmoe_b200 import ops
    c, t = _layer(N, 128, 32, E, 64, "bf16", N + E)
    x2d, wa, wb = _dev(t["x"].reshape(N, c.d)), _dev(t["wa"]), _dev(t["wb"])
    w1, b1, w2 = _dev(t["w1"]), _dev(t["b1"]), _dev(t["w2"])
    wsp = ops.Workspace.allocate(N, E, "cuda")
    rp, ep = ops.prepack_router(wa, wb), ops.prepack_experts(w1, b1, w2)
    for tau in (0.3, 1.0):
        out = torch.full((N, c.d), float("nan"), dtype=torch.bfloat16, device="cuda")
        rt = torch.empty(N, E, dtype=torch.bfloat16, device="cuda")
        ops.moe_forward(x2d, wa, wb, tau, w1, b1, w2, "relu", out, wsp, router_packed=rp,
                        last_bias=_dev(t["last_bias"].reshape(-1)), experts_packed=ep, routing_out=rt)
        wsp.check_status()
        m = O.unpack_mask(wsp.mask_bits[:N].cpu().numpy().view(np.uint32), E)
        assert torch.equal(rt.cpu() > 0, m)
        off, idx = _lists(wsp, E)
        roff, ridx = O.expert_token_lists(m)
        assert np.array_equal(off, np.asarray(roff)) and np.array_equal(idx, np.asarray(ridx))
        ex = O.experts_ffn_exact(t["x"].reshape(N, c.d), m, t["w1"], t["b1"], t["w2"])
        slack = max(1.0, m.sum(1).max().item() ** 0.5 / 2)      # one rounding per added expert
        assert O.rel_err(out.cpu().float(), ex + t["last_bias"].double()) <= TOL["bf16"] * slack


@pytest.mark.parametrize("E", [1, 2, 3])
def test_counts_table_of_few_experts_stays_in_the_workspace(E):
    from d2dmoe_b200 import ops
    N, d = 50432, 64
    c, t = _layer(N, d, 16, E, 16, "bf16", E)
    wsp = ops.Workspace.allocate(N, E, "cuda")
    need = ops.workspace_bytes(N, E)
    whole = torch.full((need + 65536,), 0xA5, dtype=torch.uint8, device="cuda")
    wsp.ws = whole[:need]
    x2d, wa, wb = _dev(t["x"].reshape(N, d)), _dev(t["wa"]), _dev(t["wb"])
    w1, b1, w2 = _dev(t["w1"]), _dev(t["b1"]), _dev(t["w2"])
    out = torch.empty(N, d, dtype=torch.bfloat16, device="cuda")
    ops.moe_forward(x2d, wa, wb, 0.3, w1, b1, w2, "relu", out, wsp,
                    router_packed=ops.prepack_router(wa, wb),
                    experts_packed=ops.prepack_experts(w1, b1, w2))
    off, idx = _lists(wsp, E)
    ops.compact(wsp, N, E)
    wsp.check_status()
    assert bool((whole[need:] == 0xA5).all())
    m = O.unpack_mask(wsp.mask_bits[:N].cpu().numpy().view(np.uint32), E)
    roff, ridx = O.expert_token_lists(m)
    for o, i in ((off, idx), _lists(wsp, E)):
        assert np.array_equal(o, np.asarray(roff)) and np.array_equal(i, np.asarray(ridx))


def test_lists_after_a_router_that_gave_up_stay_in_bounds():
    """The scatter kernel then meets a counts table that is not the mask's."""
    from d2dmoe_b200 import _capi, ops
    N, d, E = 2000, 256, 24
    c, t = _layer(N, d, 32, E, 64, "bf16", 3)
    wsp = ops.Workspace.allocate(N, E, "cuda")
    whole = torch.full((3 * N * E,), -1, dtype=torch.int32, device="cuda")
    wsp.token_idx = whole[N * E: 2 * N * E]
    x2d, wa, wb = _dev(t["x"].reshape(N, d)), _dev(t["wa"]), _dev(t["wb"])
    w1, b1, w2 = _dev(t["w1"]), _dev(t["b1"]), _dev(t["w2"])
    rp, ep = ops.prepack_router(wa, wb), ops.prepack_experts(w1, b1, w2)
    out = torch.empty(N, d, dtype=torch.bfloat16, device="cuda")
    for fill in (0xFF, 0x80, 0x01):
        wsp.ws.fill_(fill)
        wsp.mask_bits.fill_(-1)
        try:
            assert _capi.lib.d2d_debug_configure(12, 1) == 0
            ops.moe_forward(x2d, wa, wb, 0.3, w1, b1, w2, "relu", out, wsp, router_packed=rp,
                            experts_packed=ep)
            torch.cuda.synchronize()
        finally:
            _capi.lib.d2d_debug_configure(0, 0)
        with pytest.raises(_capi.D2DError, match="TIMEOUT"):
            wsp.check_status()
        assert bool((whole[: N * E] == -1).all()) and bool((whole[2 * N * E:] == -1).all())


@pytest.mark.parametrize("dtype,glu,norms", [("fp32", False, False), ("fp32", True, False),
                                             ("fp32", False, True), ("bf16", False, False)])
@pytest.mark.parametrize("e,value", [(0, -40), (2, 1 << 30), (2, -7), (3, 8 * 4 + 1), (4, 1 << 30)])
def test_offsets_out_of_range_drop_their_lists(dtype, glu, norms, e, value):
    """Reported through the status word; the lists on either side of the bad offset are skipped."""
    from d2dmoe_b200 import _capi, ops
    N, d, H, E = 8, 64, 32, 4
    c, t = _layer(N, d, H, E, 16, dtype, 5, "relu", glu)
    m = torch.ones(N, E, dtype=torch.bool)
    wsp = ops.Workspace.allocate(N, E, "cuda")
    off = torch.arange(E + 1, dtype=torch.int32) * N
    off[e] = value
    wsp.offsets.copy_(off)
    wsp.token_idx.copy_(torch.arange(N, dtype=torch.int32).repeat(E))
    m[:, [i for i in range(E) if off[i] < 0 or off[i + 1] < off[i] or off[i + 1] > N * E]] = False
    w1, b1, w2, wu = (_dev(t.get(k)) for k in ("w1", "b1", "w2", "w_up"))
    b1 = None if glu else b1
    out = torch.empty(N, d, dtype=c.torch_dtype, device="cuda")
    kw = dict(norms=torch.empty(E, N, device="cuda")) if norms else {}
    ops.experts_ffn(_dev(t["x"].reshape(N, d)), wsp, w1, b1, w2, "relu", out, w_up=wu,
                    packed=ops.prepack_experts(w1, b1, w2, wu), **kw)
    with pytest.raises(_capi.D2DError, match="INDEX_RANGE"):
        wsp.check_status()
    ex = O.experts_ffn_exact(t["x"].reshape(N, d), m, t["w1"], None if glu else t["b1"], t["w2"], "relu",
                             t.get("w_up") if glu else None)
    # one rounding per added expert
    assert O.rel_err(out.cpu().float(), ex) <= TOL[dtype]


@pytest.mark.parametrize("limit", [8, 12])
@pytest.mark.parametrize("form,N,d,H,E,R,glu", [
    ("short", 197, 256, 64, 16, 64, False), ("short", 64, 2048, 128, 32, 64, True),
    ("short", 500, 128, 32, 9, 64, False), ("long", 2000, 256, 64, 16, 64, False),
    ("long", 2000, 128, 128, 5, 64, True), ("norms", 700, 256, 64, 6, 64, False),
    ("router", 2000, 768, 32, 24, 128, False), ("router", 2000, 256, 32, 100, 256, False),
    ("cluster", 300, 2048, 32, 24, 256, False)])
def test_every_form_gives_up_and_the_next_call_is_clean(form, N, d, H, E, R, glu, limit):
    """A slice of weights that never arrives: each role leaves as whole warps, the launch ends and
    reports, and the same call right afterwards gives what it gave before."""
    from d2dmoe_b200 import _capi, ops
    c, t = _layer(N, d, H, E, R, "bf16", N + d, "relu", glu)
    x2d, wa, wb = _dev(t["x"].reshape(N, d)), _dev(t["wa"]), _dev(t["wb"])
    w1, b1, w2, wu = (_dev(t.get(k)) for k in ("w1", "b1", "w2", "w_up"))
    b1 = None if glu else b1
    wsp = ops.Workspace.allocate(N, E, "cuda")
    out = torch.empty(N, d, dtype=torch.bfloat16, device="cuda")
    if form in ("router", "cluster"):
        packed, lb = ops.prepack_router(wa, wb), _dev(t["last_bias"].reshape(-1))

        def call():
            ops.router_mask(x2d, wa, wb, 0.3, wsp, packed=packed, out_init=out, last_bias=lb)
            return wsp.mask_bits[:N].clone(), out.clone()
    else:
        m = torch.rand(N, E, generator=_gen(N)) < (0.02 if E > 16 else 0.1)
        wsp.mask_bits[:N].copy_(torch.from_numpy(O.pack_mask(m).view(np.int32)).cuda())
        ops.compact(wsp, N, E)
        packed = ops.prepack_experts(w1, b1, w2, wu)
        kw = dict(norms=torch.empty(E, N, dtype=torch.bfloat16, device="cuda")) if form == "norms" else {}

        def call():
            ops.experts_ffn(x2d, wsp, w1, b1, w2, "relu", out, w_up=wu, packed=packed, **kw)
            return (out.clone(),)
    ref = call()
    wsp.check_status()
    try:
        assert _capi.lib.d2d_debug_configure(limit, 1) == 0
        call()
        torch.cuda.synchronize()                     # returns
        with pytest.raises(_capi.D2DError, match="TIMEOUT"):
            wsp.check_status()
    finally:
        _capi.lib.d2d_debug_configure(0, 0)
    out.fill_(float("nan"))
    got = call()
    wsp.check_status()
    for a, b in zip(got, ref):
        if a.dtype == torch.int32:
            assert torch.equal(a, b)
        else:      # the order of the adds is free: one rounding each
            assert O.rel_err(a.float().cpu(), b.float().cpu()) <= TOL["bf16"]


U = 2.0 ** -8          # bf16 holds 8 bits: a rounding changes a value by at most this share of it


def _magnitudes(x2d, m, w1, b1, w2):
    """Per token and column: sum over its experts of |h W2| and of (|x W1| + |b1|) |W2|, in fp32."""
    S, A = torch.zeros_like(x2d, dtype=torch.float32), torch.zeros_like(x2d, dtype=torch.float32)
    x, m = x2d.float(), m.to(x2d.device)
    for e in range(w1.shape[0]):
        a, b, w = x @ w1[e].float(), b1[e].float(), w2[e].float()
        S += m[:, e : e + 1] * ((a + b).relu() @ w).abs()
        A += m[:, e : e + 1] * ((a.abs() + b.abs()) @ w.abs())
    return S, A


# N: tiles past the lists' cluster (1024 tokens) to more than one look at the table (96 tiles), ragged
# ends; E: one to eight 16-cell groups of counts; tau: a token in a hundred to nearly every one
@pytest.mark.parametrize("N,E,tau", [(1025, 1, 0.3), (1153, 5, 1.0), (1151, 24, 0.2), (2049, 33, 0.9), (5000, 64, 0.02),
                                     (12801, 97, 0.1), (20011, 128, 0.0), (20000, 16, 0.6), (1025, 8, 0.7), (9001, 40, 0.2)])
def test_lists_made_by_the_expert_kernel(N, E, tau):
    """Lists and offsets of a long call, from the table that the router (or the rule on given scores of whole
    16-byte rows, some of them NaN) leaves, against those of the scatter kernel, which a workspace without room
    for the table gets.  The number of launches tells that the two arms are the two forms."""
    from d2dmoe_b200 import _capi, ops
    d, H, R = 64, 16, 16
    c, t = _layer(N, d, H, E, R, "bf16", N + E)
    x2d, wa, wb = _dev(t["x"].reshape(N, d)), _dev(t["wa"]), _dev(t["wb"])
    w1, b1, w2 = _dev(t["w1"]), _dev(t["b1"]), _dev(t["w2"])
    rp, ep = ops.prepack_router(wa, wb), ops.prepack_experts(w1, b1, w2)
    scores = torch.rand(N, E, generator=_gen(N), dtype=torch.float32).to(torch.bfloat16).cuda()
    scores[5::97] = float("nan")
    for given in (None, scores) if E % 8 == 0 and E <= 64 else (None,):
        got = []
        for room in (True, False):
            wsp = ops.Workspace.allocate(N, E, "cuda")
            if not room:
                wsp.ws = wsp.ws[: -(-N // 128) * max(16, 1 << (E - 1).bit_length(), 4 * E) + 4 * E]
            wsp.token_idx.fill_(-1)
            out = torch.empty(N, d, dtype=torch.bfloat16, device="cuda")
            ops.moe_forward(x2d, None if given is not None else wa, None if given is not None else wb, tau, w1,
                            b1, w2, "relu", out, wsp, scores=given, experts_packed=ep,
                            router_packed=None if given is not None else rp)
            assert _capi.lib.d2d_last_forward_launches() == (2 if room else 3)
            wsp.check_status()
            got.append((_lists(wsp, E), out, wsp.mask_bits[:N].clone(), wsp.token_idx.clone()))
        (l0, o0, m0, i0), (l1, o1, m1, i1) = got
        assert torch.equal(m0, m1) and np.array_equal(l0[0], l1[0]) and np.array_equal(l0[1], l1[1])
        assert torch.equal(i0, i1)                       # nothing behind the lists either
        m = O.unpack_mask(m0.cpu().numpy().view(np.uint32), E)
        roff, ridx = O.expert_token_lists(m)
        assert np.array_equal(l0[0], np.asarray(roff)) and np.array_equal(l0[1], np.asarray(ridx))
        if given is not None:
            assert not m[5::97].any() and m[:5].any(1).all()
        # Both arms add the same bf16 contributions in an order of their own: each of a token's k - 1 adds rounds by
        # U of a running sum, which is at most S and what the contributions are rounded by (4 times U
        # of A, see below).  One add: equal.
        S, A = _magnitudes(x2d, m, w1, b1, w2)
        k = m.sum(1, keepdim=True).cuda()
        lim = 1.02 * 2 * (k - 1).clamp(min=0) * U * (S + 4 * U * A)
        diff = (o0.float() - o1.float()).abs()
        assert bool((diff <= lim).all()), ((diff - lim).max(), (diff * (k == 1)).max())
        # against the exact sum: x W1, its sum with b1 and the hidden value are rounded (3 times U of A at
        # most), then each contribution and each add (U of S, at most A)
        ex = O.experts_ffn_exact(x2d.cpu(), m, w1.cpu(), b1.cpu(), w2.cpu(), "relu").cuda()
        assert bool(((o0.double() - ex).abs() <= 1.02 * (3 + 1 + k) * U * A).all())


@pytest.mark.parametrize("N,launches", [(511 * 15 * 128, 2), (511 * 15 * 128 + 1, 3)])
def test_lists_of_the_longest_calls(N, launches):
    """Every expert on every token: the 16-bit sums of the table's fifteen parts at their largest (511 tiles of
    128 tokens), and the first call that is too long for them."""
    from d2dmoe_b200 import _capi, ops
    d, H, E, R = 64, 16, 8, 16
    c, t = _layer(64, d, H, E, R, "bf16", 3)
    x2d = _dev(t["x"].reshape(64, d)).repeat(-(-N // 64), 1)[:N].contiguous()
    wa, wb, w1, b1, w2 = (_dev(t[n]) for n in ("wa", "wb", "w1", "b1", "w2"))
    wsp, out = ops.Workspace.allocate(N, E, "cuda"), torch.empty_like(x2d)
    wsp.token_idx.fill_(-1)
    ops.moe_forward(x2d, wa, wb, 1.0, w1, b1, w2, "relu", out, wsp, experts_packed=ops.prepack_experts(w1, b1, w2),
                    router_packed=ops.prepack_router(wa, wb))
    assert _capi.lib.d2d_last_forward_launches() == launches
    wsp.check_status()
    each = torch.arange(N, dtype=torch.int32, device="cuda")
    assert torch.equal(wsp.offsets, torch.arange(E + 1, dtype=torch.int32, device="cuda") * N)
    assert torch.equal(wsp.token_idx.view(E, N), each.expand(E, N))
    m = torch.ones(64, E, dtype=torch.bool)
    ex = O.experts_ffn_exact(t["x"].reshape(64, d), m, t["w1"], t["b1"], t["w2"], "relu").cuda()
    _, A = _magnitudes(x2d[:64], m, w1, b1, w2)
    lim = (1.02 * (4 + E) * U * A).repeat(-(-N // 64), 1)[:N]        # as above
    assert bool(((out.double() - ex.repeat(-(-N // 64), 1)[:N]).abs() <= lim).all())


@pytest.mark.parametrize("N,E,glu", [(2000, 16, False), (5000, 24, True)])
def test_layer_gives_up_over_a_table_that_is_not_the_masks(N, E, glu):
    """Router and experts both miss a slice of weights, and where the router leaves nothing the table holds more
    tokens than there are: the call ends and reports, nothing is written past the lists, the next one is right."""
    from d2dmoe_b200 import _capi, ops
    d, H, R = 256, 64, 64
    c, t = _layer(N, d, H, E, R, "bf16", N, "relu", glu)
    x2d, wa, wb = _dev(t["x"].reshape(N, d)), _dev(t["wa"]), _dev(t["wb"])
    w1, b1, w2, wu = (_dev(t.get(k)) for k in ("w1", "b1", "w2", "w_up"))
    b1 = None if glu else b1
    rp, ep = ops.prepack_router(wa, wb), ops.prepack_experts(w1, b1, w2, wu)
    wsp = ops.Workspace.allocate(N, E, "cuda")
    whole = torch.full((2 * N * E,), -1, dtype=torch.int32, device="cuda")
    wsp.token_idx = whole[: N * E]
    out = torch.empty(N, d, dtype=torch.bfloat16, device="cuda")

    def call():
        ops.moe_forward(x2d, wa, wb, 0.2, w1, b1, w2, "relu", out, wsp, w_up=wu, experts_packed=ep, router_packed=rp)
        assert _capi.lib.d2d_last_forward_launches() == 2
    call()
    wsp.check_status()
    ref, lists = out.clone(), _lists(wsp, E)
    wsp.ws.fill_(255)
    try:
        assert _capi.lib.d2d_debug_configure(12, 1) == 0
        call()
        torch.cuda.synchronize()                     # returns
    finally:
        _capi.lib.d2d_debug_configure(0, 0)
    with pytest.raises(_capi.D2DError, match="TIMEOUT"):
        wsp.check_status()
    assert bool((whole[N * E :] == -1).all())
    out.fill_(float("nan"))
    call()
    wsp.check_status()
    got = _lists(wsp, E)
    assert np.array_equal(got[0], lists[0]) and np.array_equal(got[1], lists[1])
    assert O.rel_err(out.float().cpu(), ref.float().cpu()) <= TOL["bf16"]      # (the order of the adds is free)


@pytest.mark.parametrize("bias", [True, False])
@pytest.mark.parametrize("N,d", [(1, 64), (129, 768), (1025, 512), (18945, 768), (20011, 128)])
def test_initial_rows_of_a_residual_layer(N, d, bias):
    """x + last_bias, one rounding, exactly: the rows come out of the stages of the router's first product (one
    stage to several laps of the ring, one tile to two per CTA, a last tile of one row)."""
    from d2dmoe_b200 import ops
    E, R = 12, 128
    c, t = _layer(N, d, 16, E, R, "bf16", N + d)
    x2d, wa, wb = _dev(t["x"].reshape(N, d)), _dev(t["wa"]), _dev(t["wb"])
    lb = _dev(t["last_bias"].reshape(-1)) if bias else None
    packed, wsp = ops.prepack_router(wa, wb), ops.Workspace.allocate(N, E, "cuda")
    for _ in range(8):
        out = torch.full((N, d), float("nan"), dtype=torch.bfloat16, device="cuda")
        ops.router_mask(x2d, wa, wb, 0.3, wsp, packed=packed, out_init=out, last_bias=lb, add_residual=True)
        wsp.check_status()
        assert torch.equal(out, x2d + lb if bias else x2d + 0)


@pytest.mark.parametrize("bias", [True, False])
@pytest.mark.parametrize("N,d", [(1, 64), (127, 768), (130, 2048), (1024, 64), (1025, 320), (14208, 64), (14209, 64)])
def test_initial_rows_by_other_blocks(N, d, bias):
    """last_bias in every row, exactly, of the router's own call (by the blocks that have no tile up to 18 tiles: one
    tile, one cluster of eight, more), and the layer on either side of its line at 111 tiles."""
    from d2dmoe_b200 import ops
    E, R = 3, 16
    c, t = _layer(N, d, 16, E, R, "bf16", N + d)
    x2d, wa, wb = _dev(t["x"].reshape(N, d)), _dev(t["wa"]), _dev(t["wb"])
    w1, b1, w2 = _dev(t["w1"]), _dev(t["b1"]), _dev(t["w2"])
    lb = _dev(t["last_bias"].reshape(-1)) if bias else None
    packed, wsp = ops.prepack_router(wa, wb), ops.Workspace.allocate(N, E, "cuda")
    out = torch.full((N, d), float("nan"), dtype=torch.bfloat16, device="cuda")
    ops.router_mask(x2d, wa, wb, 0.3, wsp, packed=packed, out_init=out, last_bias=lb)
    wsp.check_status()
    assert torch.equal(out, lb.expand(N, d) if bias else torch.zeros_like(out))
    for residual in (False, True):
        out.fill_(float("nan"))
        ops.moe_forward(x2d, wa, wb, 0.3, w1, b1, w2, "relu", out, wsp, last_bias=lb, router_packed=packed,
                        experts_packed=ops.prepack_experts(w1, b1, w2), add_residual=residual)
        wsp.check_status()
        m = O.unpack_mask(wsp.mask_bits[:N].cpu().numpy().view(np.uint32), E)
        ex = O.experts_ffn_exact(t["x"].reshape(N, d), m, t["w1"], t["b1"], t["w2"])
        ex = ex + (t["last_bias"].double() if bias else 0.0) + (t["x"].reshape(N, d).double() if residual else 0.0)
        assert O.rel_err(out.cpu().float(), ex) <= TOL["bf16"]


@pytest.mark.parametrize("dtype,E", [("bf16", 24), ("fp32", 8)])
@pytest.mark.parametrize("N", [1, 127, 1024, 1025, 18944, 18945])
def test_initial_rows_beside_given_scores(N, dtype, E):
    """The same where the scores are given (one tile, one cluster of eight, more; either side of the rule's line at
    148 tiles)."""
    from d2dmoe_b200 import ops
    d = 64
    c, t = _layer(N, d, 16, E, 16, dtype, N + E)
    dt = t["x"].dtype
    x2d, w1, b1, w2 = _dev(t["x"].reshape(N, d)), _dev(t["w1"]), _dev(t["b1"]), _dev(t["w2"])
    lb = _dev(t["last_bias"].reshape(-1))
    scores = torch.rand(N, E, generator=_gen(N)).to(dt)
    packed = ops.prepack_experts(w1, b1, w2) if dtype == "bf16" else None
    wsp = ops.Workspace.allocate(N, E, "cuda")
    m = O.dynk_max_mask(scores, 0.1)
    ex = O.experts_ffn_exact(t["x"].reshape(N, d), m, t["w1"], t["b1"], t["w2"]) + t["last_bias"].double()
    for residual in (False, True):
        out = torch.full((N, d), float("nan"), dtype=dt, device="cuda")
        ops.moe_forward(x2d, None, None, 0.1, w1, b1, w2, "relu", out, wsp, last_bias=lb, scores=_dev(scores),
                        experts_packed=packed, add_residual=residual)
        wsp.check_status()
        assert torch.equal(O.unpack_mask(wsp.mask_bits[:N].cpu().numpy().view(np.uint32), E), m)
        want = ex + (t["x"].reshape(N, d).double() if residual else 0.0)
        assert O.rel_err(out.cpu().float(), want) <= TOL[dtype]


@pytest.mark.parametrize("N,resid", [(1100, False), (2000, True), (20011, False)])
def test_waits_begin_when_the_previous_kernel_is_over(N, resid):
    """A router call behind one that takes some 80 ms to give up: its bounded waits (a few ms here) are for its own
    copies and products, not for the kernel in front of it, whose blocks it may start beside."""
    from d2dmoe_b200 import _capi, ops
    d, E, R = 256, 24, 64
    c, t = _layer(N, d, 32, E, R, "bf16", N)
    x2d, wa, wb = _dev(t["x"].reshape(N, d)), _dev(t["wa"]), _dev(t["wb"])
    packed = ops.prepack_router(wa, wb)
    first, then = ops.Workspace.allocate(N, E, "cuda"), ops.Workspace.allocate(N, E, "cuda")
    out = torch.empty(N, d, dtype=torch.bfloat16, device="cuda")

    def call(wsp):
        ops.router_mask(x2d, wa, wb, 0.3, wsp, packed=packed, out_init=out, add_residual=resid)
    call(then)
    ref = then.mask_bits[:N].clone()
    then.check_status()
    try:
        assert _capi.lib.d2d_debug_configure(18, 1) == 0
        call(first)
        assert _capi.lib.d2d_debug_configure(14, 0) == 0
        call(then)
        torch.cuda.synchronize()
    finally:
        _capi.lib.d2d_debug_configure(0, 0)
    with pytest.raises(_capi.D2DError, match="TIMEOUT"):
        first.check_status()
    then.check_status()
    assert torch.equal(then.mask_bits[:N], ref)


@pytest.mark.gpu
@pytest.mark.parametrize("mode,k,E,N", [("topk", 2, 5, 95), ("topk", 2, 5, 999), ("topk", 4, 5, 500), ("all", 5, 5, 399),
                                        ("all", 5, 5, 400), ("dynk", 0, 5, 961), ("dynk_max", 0, 5, 959),
                                        ("dynk_max", 0, 5, 960), ("topk", 2, 24, 1463), ("topk", 2, 24, 1464),
                                        ("all", 24, 24, 240), ("all", 24, 24, 241), ("all", 24, 24, 289)])
def test_fp32_items_of_several_ragged_lists(mode, k, E, N):
    """Item sizes of 16 and of 32 rows over several experts with ragged lists, on either side of the
    lines of the rule that chooses between them (mean list of 288 or 400 rows; rounds of CTAs)."""
    import d2dmoe_b200 as D
    d, H = 132, 100
    c, t = _layer(N, d, H, E, 36, "fp32", N + k)
    moe = D.MoeficationMoE("m", d, E, True, H, torch.nn.ReLU)
    moe.router = D.MoeficationRouter(d, E, width=36, depth=2, bias=False, activation="relu", output_activation="abs")
    moe.load_state_dict({"experts.w1": t["w1"], "experts.b1": t["b1"], "experts.w2": t["w2"], "last_bias": t["last_bias"],
                         "router.layers.0.weight": t["wa"], "router.layers.2.weight": t["wb"]})
    moe = moe.cuda().eval()
    moe.forward_mode, moe.k, moe.tau = mode, k, 0.6
    with torch.no_grad():
        out, gating = moe(_dev(t["x"]))
    m = gating["m"][0].reshape(N, E).cpu() > 0
    if mode in ("topk", "all"):
        assert (m.sum(1) == (k if mode == "topk" else E)).all()
    ex = O.experts_ffn_exact(t["x"].reshape(N, d), m, t["w1"], t["b1"], t["w2"]) + t["last_bias"].double()
    assert O.rel_err(out.reshape(N, d).cpu(), ex) <= TOL["fp32"]


@pytest.mark.parametrize("tau,N", [(0.02, 50 * 128), (0.02, 50 * 128 + 1), (0.0, 44 * 128), (0.0, 44 * 128 + 1),
                                   (1.0, 111 * 128), (1.0, 111 * 128 + 1), (-1.0, 20), (-1.0, 1024), (-1.0, 1025)])
def test_who_writes_initial_rows_by_the_threshold(tau, N):
    """The blocks without a tile write them up to a line that follows the threshold (no share of the tokens expected
    to keep several experts, a small one, all; a threshold above the maximum, where no blocks help): the layer on either
    side of it, on a device of 148 SMs."""
    from d2dmoe_b200 import ops
    E, R, d = 3, 16, 64
    c, t = _layer(N, d, 16, E, R, "bf16", N)
    x2d, wa, wb = _dev(t["x"].reshape(N, d)), _dev(t["wa"]), _dev(t["wb"])
    w1, b1, w2, lb = _dev(t["w1"]), _dev(t["b1"]), _dev(t["w2"]), _dev(t["last_bias"].reshape(-1))
    wsp = ops.Workspace.allocate(N, E, "cuda")
    out = torch.full((N, d), float("nan"), dtype=torch.bfloat16, device="cuda")
    ops.moe_forward(x2d, wa, wb, tau, w1, b1, w2, "relu", out, wsp, last_bias=lb, router_packed=ops.prepack_router(wa, wb),
                    experts_packed=ops.prepack_experts(w1, b1, w2))
    wsp.check_status()
    m = O.unpack_mask(wsp.mask_bits[:N].cpu().numpy().view(np.uint32), E)
    assert (m.sum(1) == E).all() if tau == 1.0 else tau < 0 or (m.sum(1) >= 1).all()
    ex = O.experts_ffn_exact(t["x"].reshape(N, d), m, t["w1"], t["b1"], t["w2"]) + t["last_bias"].double()
    assert O.rel_err(out.cpu().float(), ex) <= TOL["bf16"]


@pytest.mark.parametrize("N", [18 * 128, 18 * 128 + 1, 74 * 128, 74 * 128 + 1])
def test_initial_rows_at_the_other_lines(N):
    """Every row from last_bias (ranked rules, the router's own call: 18 tiles) or with the layer's input added (74
    tiles): the rows themselves, exactly, and top-k and dynk layers, on a device of 148 SMs."""
    from d2dmoe_b200 import ops
    import d2dmoe_b200 as D
    E, R, d, H = 4, 16, 64, 16
    c, t = _layer(N, d, H, E, R, "bf16", N)
    x2d, wa, wb, lb = _dev(t["x"].reshape(N, d)), _dev(t["wa"]), _dev(t["wb"]), _dev(t["last_bias"].reshape(-1))
    packed, wsp = ops.prepack_router(wa, wb), ops.Workspace.allocate(N, E, "cuda")
    for residual in (False, True):
        out = torch.full((N, d), float("nan"), dtype=torch.bfloat16, device="cuda")
        ops.router_mask(x2d, wa, wb, 0.3, wsp, packed=packed, out_init=out, last_bias=lb, add_residual=residual)
        wsp.check_status()
        assert torch.equal(out, x2d + lb if residual else lb.expand(N, d))
        for mode, k in (("topk", 1), ("topk", 3), ("dynk", 0)):
            moe = D.MoeficationMoE("m", d, E, True, H, torch.nn.ReLU, add_residual_connection=residual)
            moe.router = D.MoeficationRouter(d, E, width=R, depth=2, bias=False, activation="relu", output_activation="abs")
            moe = moe.bfloat16()
            moe.load_state_dict({"experts.w1": t["w1"], "experts.b1": t["b1"], "experts.w2": t["w2"],
                                 "last_bias": t["last_bias"], "router.layers.0.weight": t["wa"],
                                 "router.layers.2.weight": t["wb"]})
            moe = moe.cuda().eval()
            moe.forward_mode, moe.k, moe.tau = mode, k, 0.6
            with torch.no_grad():
                got, gating = moe(_dev(t["x"]))
            m = gating["m"][0].reshape(N, E).cpu() > 0
            ex = O.experts_ffn_exact(t["x"].reshape(N, d), m, t["w1"], t["b1"], t["w2"]) + t["last_bias"].double()
            ex = ex + (t["x"].reshape(N, d).double() if residual else 0.0)
            assert O.rel_err(got.reshape(N, d).cpu().float(), ex) <= TOL["bf16"], (mode, k, residual)


@pytest.mark.parametrize("mode,k", [("topk", 1), ("topk", 3), ("dynk", 0)])
@pytest.mark.parametrize("N", [1025, 18944, 18945])
def test_initial_rows_beside_given_scores_of_ranked_rules(N, mode, k):
    """The same for top-k and dynk on given scores: more than one cluster, either side of 148 tiles."""
    import d2dmoe_b200 as D
    E, d, H = 24, 64, 16
    c, t = _layer(N, d, H, E, 16, "bf16", N)
    scores = torch.rand(1, N, E, generator=_gen(N)).bfloat16()
    sd = _dev(scores)

    class Given(torch.nn.Module):
        def forward(self, x):
            return sd

    for residual in (False, True):
        moe = D.MoeficationMoE("m", d, E, True, H, torch.nn.ReLU, add_residual_connection=residual).bfloat16()
        moe.load_state_dict({"experts.w1": t["w1"], "experts.b1": t["b1"], "experts.w2": t["w2"], "last_bias": t["last_bias"]},
                            strict=False)
        moe = moe.cuda().eval()
        moe.router = Given()
        moe.forward_mode, moe.k, moe.tau = mode, k, 0.2
        with torch.no_grad():
            got, gating = moe(_dev(t["x"]))
        m = gating["m"][0].reshape(N, E).cpu() > 0
        if mode == "topk":
            # (equal scores may be taken in either order: what was taken is no less than what was left)
            s = scores.reshape(N, E).float()
            assert (m.sum(1) == k).all()
            assert (s.masked_fill(~m, 2.0).amin(1) >= s.masked_fill(m, -1.0).amax(1)).all()
        ex = O.experts_ffn_exact(t["x"].reshape(N, d), m, t["w1"], t["b1"], t["w2"]) + t["last_bias"].double()
        ex = ex + (t["x"].reshape(N, d).double() if residual else 0.0)
        assert O.rel_err(got.reshape(N, d).cpu().float(), ex) <= TOL["bf16"], residual
