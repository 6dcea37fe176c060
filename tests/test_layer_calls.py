"""Calls of the layer around its kept facts: what a plan, a workspace or a staging buffer is made
from may change between two calls, on another stream or in another thread."""
import copy

import pytest
import torch

from helpers import C, O, TOL

pytestmark = pytest.mark.gpu


def _moe(c, t, experts=None, router=None):
    import d2dmoe_b200 as D
    moe = D.MoeficationMoE(c.name, c.d, c.E, True, c.H, torch.nn.ReLU)
    if experts is not None:
        moe.experts = experts(c.d, c.E, 2, c.H, "without_last", torch.nn.ReLU)
    moe.router = (router or D.MoeficationRouter)(c.d, c.E, width=c.R, depth=2, bias=False,
                                                 activation="relu", output_activation="abs")
    moe = moe.to(c.torch_dtype)
    moe.load_state_dict({"experts.w1": t["w1"], "experts.b1": t["b1"], "experts.w2": t["w2"],
                         "last_bias": t["last_bias"], "router.layers.0.weight": t["wa"],
                         "router.layers.2.weight": t["wb"]})
    moe = moe.cuda().eval()
    moe.forward_mode, moe.tau = "dynk_max", c.tau
    return moe


def _case(N=197, dtype="bf16", B=1, **kw):
    c = C.LayerCase("calls", B, N, 128, 64, 8, R=64, tau=0.3, dtype=dtype, seed=N, **kw)
    return c, C.make_tensors(c)


def _same(moe, x, call="forward"):
    """The call's result against a layer that has never been called before."""
    fresh = copy.deepcopy(moe)
    want, _ = fresh(x)
    if call == "forward":
        got, _ = moe(x)
    elif call == "block":
        norm = torch.nn.LayerNorm(x.size(-1)).to(x)
        got, _ = moe.forward_block(x, norm)
        want, _ = fresh.forward_block(x, norm)
    else:
        got = moe.forward_host(x.cpu().pin_memory()).cuda()
    return O.rel_err(got.float().cpu(), want.float().cpu()) <= TOL["bf16"]


@pytest.mark.parametrize("call", ["forward", "block", "host"])
@pytest.mark.parametrize("which", ["experts", "router"])
def test_invalidate_packed_reaches_every_call(which, call):
    """Writes through .data leave the version counter alone; invalidate_packed() announces them."""
    c, t = _case()
    moe, x = _moe(c, t), t["x"].cuda()
    assert _same(moe, x, call)
    p = moe.experts.w2 if which == "experts" else moe.router.layers[0].weight
    p.data.copy_(torch.roll(p.detach(), 1, 0 if which == "experts" else 1) * 3.0)
    getattr(moe, which).invalidate_packed()
    assert _same(moe, x, call)


def test_activation_and_bias_are_read_at_each_call():
    c, t = _case()
    moe, x = _moe(c, t), t["x"].cuda()
    assert _same(moe, x)
    moe.experts.activation_str = "leaky_relu"
    moe.experts.b1.data.sub_(4.0)                # (hidden values that the two activations tell apart)
    moe.experts.invalidate_packed()
    assert _same(moe, x)
    moe.last_bias.data.add_(5.0)
    assert _same(moe, x)
    moe.bias = False
    assert _same(moe, x)


@pytest.mark.parametrize("dtype", ["bf16", "fp32"])
def test_weights_that_are_no_parameters_are_read_at_each_call(dtype):
    """Pruning replaces the parameter by a plain attribute that a hook writes anew."""
    from torch.nn.utils import prune
    c, t = _case(dtype=dtype)
    moe, plain, x = _moe(c, t), _moe(c, t), t["x"].cuda()
    lin = moe.router.layers[0]
    g = torch.Generator().manual_seed(1)
    prune.custom_from_mask(lin, "weight", (torch.rand(c.R, c.d, generator=g) < 0.5).cuda())
    for _ in range(2):
        with torch.no_grad():
            lin.weight_orig.copy_(torch.roll(lin.weight_orig, 1, 1))
            moe.router(x)                        # the hook writes lin.weight
            plain.router.layers[0].weight.copy_(lin.weight)
        assert torch.equal(moe(x)[1][c.name][0], plain(x)[1][c.name][0])


def test_a_call_that_does_not_fit_keeps_the_plan(monkeypatch):
    """fp32 scores on a bf16 layer take the general path; the plan stays."""
    class Scores(torch.nn.Module):
        def forward(self, x):
            return torch.linspace(0, 1, 8, device=x.device).expand(*x.shape[:-1], 8)
    c, t = _case()
    moe, x = _moe(c, t), t["x"].cuda()
    moe.router, moe.forward_mode, moe.k = Scores(), "topk", 2
    made = []
    make = type(moe)._make_plan
    monkeypatch.setattr(type(moe), "_make_plan", lambda self: made.append(1) or make(self))
    for _ in range(3):
        out, gd = moe(x)
    assert gd[c.name][0].dtype == torch.float32 and int(gd[c.name][0][..., 6:].sum()) == 2 * c.N
    assert len(made) == 1


def test_subclasses_take_the_fused_path():
    import d2dmoe_b200 as D

    class Router(D.MoeficationRouter):
        def forward(self, x):
            raise AssertionError("'dynk_max' does not call a fusable router")

    class Experts(D.B200KernelExperts):
        pass
    c, t = _case()
    moe, x = _moe(c, t, Experts, Router), t["x"].cuda()
    plain = _moe(c, t)
    for call in (lambda m: m(x), lambda m: m.forward_block(x, torch.nn.LayerNorm(c.d).to(x))):
        got, want = call(moe), call(plain)
        assert torch.equal(got[1][c.name][0], want[1][c.name][0])
        assert O.rel_err(got[0].float().cpu(), want[0].float().cpu()) <= TOL["bf16"]
    assert moe._plan.handle is not None


@pytest.mark.parametrize("how", ["layer", "bias", "forward", "override", "autocast"])
def test_ranked_rules_call_a_router_that_was_changed(how):
    """'topk' and 'dynk' rank what the router module returns."""
    c, t = _case(dtype="fp32" if how == "autocast" else "bf16")
    moe, x = _moe(c, t), t["x"].cuda()
    moe.forward_mode, moe.k = "topk", 3
    r = moe.router
    if how == "layer":
        r.layers[1] = torch.nn.Tanh()
    elif how == "bias":
        r.layers[2].bias = torch.nn.Parameter(torch.linspace(-9, 9, c.E, dtype=c.torch_dtype).cuda())
    elif how == "forward":
        flipped = type(r).forward
        r.forward = lambda v: 1.0 / (1.0 + flipped(r, v))
    elif how == "override":
        r.test_override_outputs_p, r.response_cache = 0.5, {}
    with torch.no_grad(), torch.autocast("cuda", torch.bfloat16, enabled=how == "autocast"):
        rt = moe(x)[1][c.name][0]
        s = r(x)
    best = torch.zeros_like(s).scatter_(-1, torch.sort(s.float(), dim=-1, descending=True, stable=True)[1][..., :3], 1)
    assert rt.dtype == s.dtype and torch.equal(rt, best)


def test_forward_host_beside_a_busy_stream():
    """sync=False: packing, workspaces and kernels depend on nothing the caller's stream is doing.
    A first call, new slice sizes (more than the cache keeps), changed weights, and forward() calls of
    the same token counts in between."""
    import d2dmoe_b200 as D
    c, t = _case(40, B=24)
    moe, plain, x = _moe(c, t), _moe(c, t), t["x"].pin_memory()
    for change in (False, True):
        if change:
            with torch.no_grad():
                moe.experts.w1.mul_(2), plain.experts.w1.mul_(2)
        want = {b: plain(x[:b].cuda())[0].cpu() for b in range(2, 25)}
        xd = {b: x[:b].cuda() for b in want}
        torch.cuda.synchronize()
        torch.cuda._sleep(100_000_000)
        got, dev = {}, {}
        for b in want:
            got[b] = torch.empty_like(x[:b]).pin_memory()
            moe.forward_host(x[:b], got[b], chunks=2, sync=False)
            dev[b] = moe(xd[(b + 1) // 2])[0] if b > 3 else None
        D.MoeficationMoE.host_synchronize()
        torch.cuda.synchronize()
        for b in want:
            assert O.rel_err(got[b].float(), want[b].float()) <= TOL["bf16"], b
            if b > 3:
                assert O.rel_err(dev[b].float().cpu(), want[(b + 1) // 2].float()) <= TOL["bf16"], b


@pytest.mark.parametrize("dtype,other", [("bf16", torch.float32), ("fp32", torch.bfloat16)])
@pytest.mark.parametrize("mode", ["dynk_max", "topk", "dynk"])
def test_scores_in_another_dtype(mode, dtype, other):
    """A router whose scores are not of x's dtype (autocast): the rule applies to them as they are."""
    class Scores(torch.nn.Module):
        def forward(self, x):
            return given
    c, t = _case(dtype=dtype)
    moe, x = _moe(c, t), t["x"].cuda()
    given = torch.exp(torch.randn(1, c.N, c.E, generator=torch.Generator().manual_seed(2))).to(other).cuda()
    moe.router, moe.forward_mode, moe.k = Scores(), mode, 2
    out, gd = moe(x)
    rt = gd[c.name][0]
    s2 = given.reshape(c.N, c.E)
    if mode == "dynk_max":
        m = O.dynk_max_mask(s2.cpu(), c.tau)
    else:
        from d2dmoe_b200 import ops
        wsp = ops.Workspace.allocate(c.N, c.E, "cuda")
        ops.mask_rule_from_scores(s2, mode, wsp, k=2, tau=c.tau)
        m = ops.expand_mask(wsp, c.N, c.E, other).cpu() > 0
    assert rt.dtype == other and torch.equal(rt.reshape(c.N, c.E).cpu() > 0, m)
    ex = O.experts_ffn_exact(t["x"].reshape(c.N, c.d), m, t["w1"], t["b1"], t["w2"])
    ex = ex + t["last_bias"].double()
    assert O.rel_err(out.reshape(c.N, c.d).cpu().float(), ex) <= TOL[dtype]


@pytest.mark.parametrize("which", ["weight", "bias"])
def test_norm_parameters_on_another_device_are_refused(which):
    c, t = _case()
    moe, x = _moe(c, t), t["x"].cuda()
    norm = torch.nn.LayerNorm(c.d).to(x)
    setattr(norm, which, torch.nn.Parameter(getattr(norm, which).detach().cpu()))
    with pytest.raises((RuntimeError, ValueError)):
        moe.forward_block(x, norm)


def test_pinned_buffers_dropped_while_the_pipeline_copies():
    """sync=False: a dropped input is still read, a dropped output still written; neither block may
    serve a new tensor meanwhile."""
    import d2dmoe_b200 as D
    from d2dmoe_b200 import moe as impl
    c, t = _case(64, B=8)
    moe = _moe(c, t)
    want = moe(t["x"].cuda())[0].cpu()
    out = moe.forward_host(t["x"].pin_memory())
    assert O.rel_err(out.float(), want.float()) <= TOL["bf16"]
    out.fill_(0.0)
    with torch.cuda.stream(impl._HOST_STREAMS[moe.experts.w1.device][0]):
        torch.cuda._sleep(200_000_000)
    x = t["x"].pin_memory()
    moe.forward_host(x, out, sync=False)
    moe.forward_host(x, torch.empty_like(x).pin_memory(), sync=False)
    del x
    new = [torch.full_like(t["x"], 7.0).pin_memory() for _ in range(4)]
    D.MoeficationMoE.host_synchronize()
    assert O.rel_err(out.float(), want.float()) <= TOL["bf16"]
    assert all(bool((v == 7.0).all()) for v in new)


def test_forward_host_keeps_its_buffers_while_another_thread_changes_them(monkeypatch):
    """A call with other slices, as another thread would make it, between the choice of the staging
    buffers and their use."""
    from types import SimpleNamespace
    from d2dmoe_b200 import moe as impl
    c, t = _case(40, B=8)
    moe, x, used = _moe(c, t), t["x"], []
    real = impl.host
    monkeypatch.setattr(impl, "host", SimpleNamespace(**{
        **vars(real), "run_host": lambda *a: used.append((tuple(a[6].shape), a[8][0].shape[0])) or True}))
    make = type(moe)._make_plan

    def between(self):
        monkeypatch.setattr(type(moe), "_make_plan", make)
        moe.forward_host(x[:2], chunks=2)
        return make(self)
    monkeypatch.setattr(type(moe), "_make_plan", between)
    moe.forward_host(x, chunks=2)
    assert used == [((2, 40, c.d), 1), ((8, 40, c.d), 4)]
