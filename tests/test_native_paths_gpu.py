"""What the native nodes of attention and block must not change: the calls that go to the autograd functions and modules
instead, what is refused, what is kept for the backward, memory and precision."""
import pytest
import torch
import torch.autograd.forward_ad as fwAD
from torch.utils._python_dispatch import TorchDispatchMode

import forgetting_transformer_b200 as fox
from forgetting_transformer_b200 import _lib, ops
from oracle import fox_oracle as orc

pytestmark = pytest.mark.gpu


def _qkvg(B=1, H=2, M=256, N=256, D=64, dtype=torch.bfloat16, seed=0):
    g = torch.Generator().manual_seed(seed)
    q, k, v = [torch.randn(B, H, t, D, generator=g).to(dtype).cuda() for t in (M, N, N)]
    return q, k, v, torch.nn.functional.logsigmoid(torch.randn(B, H, N, generator=g) + 3).cuda()


def _block(C=256, H=4, inter=512, dtype=torch.bfloat16, **kw):
    torch.manual_seed(0)
    return fox.FoxProBlock(C, H, inter, fgate_bias=2.0, **kw).cuda().to(dtype)


def _x(T=64, C=256, dtype=torch.bfloat16, seed=1, B=1):
    return torch.randn(B, T, C, generator=torch.Generator().manual_seed(seed)).to(dtype).cuda()


def _cache(blk, B=1, N=16):
    """A cache of N tokens for layer 0."""
    H, D = blk.attn.num_heads, blk.attn.head_dim
    cache, st = fox.FgateCache(), blk.attn.init_shift_state(B)
    cache.update_shift_cache(st["key_shift"], st["value_shift"], 0)
    _, k, v, g = _qkvg(B, H, N, N, D, blk.attn.q_proj.weight.dtype)
    cache.update(k, v, g, 0)
    return cache


@pytest.mark.parametrize("which", range(4))
@pytest.mark.parametrize("head_first", [True, False])
def test_forward_mode_is_refused_by_attention(which, head_first):
    """No forward derivative is built: a dual tensor raises and does not come back without its tangent."""
    args = [t if head_first else t.transpose(1, 2) for t in _qkvg()]
    with fwAD.dual_level():
        args[which] = fwAD.make_dual(args[which], torch.ones_like(args[which]))
        with pytest.raises(NotImplementedError, match="jvp"):
            fox.forgetting_attention(*args, head_first=head_first)


@pytest.mark.parametrize("T", [1, 64])
@pytest.mark.parametrize("of", ["input", "weight"])
def test_forward_mode_is_refused_by_block(T, of):
    blk, x = _block(), _x(T)
    with fwAD.dual_level(), torch.no_grad():
        if of == "input":
            x = fwAD.make_dual(x, torch.ones_like(x))
        else:
            w = blk.mlp_norm.weight.detach()
            del blk.mlp_norm.weight
            blk.mlp_norm.weight = fwAD.make_dual(w, torch.ones_like(w))
            blk.mlp_norm._parameters["weight"] = blk.mlp_norm.weight
        with pytest.raises(NotImplementedError, match="jvp"):
            blk(x, None, *((_cache(blk), 0) if T == 1 else ()))


@pytest.mark.parametrize("head_first", [True, False])
def test_traced_attention_runs_on_other_inputs(head_first):
    """torch.jit.trace records the call, not the memory its result was made in."""
    a, b = [[t if head_first else t.transpose(1, 2).contiguous() for t in _qkvg(seed=s)] for s in (1, 2)]
    f = lambda *t: fox.forgetting_attention(*t, head_first=head_first, adaptive_threshold="auto") * 1.0
    traced = torch.jit.trace(f, a, check_trace=False)
    got = traced(*b)
    assert torch.equal(got, f(*b))


@pytest.mark.parametrize("T", [1, 64])
def test_block_is_not_traced_natively(T):
    """Under torch.jit.trace the modules run one by one: their recorded operators reach the result."""
    blk, x = _block().requires_grad_(False), _x(T)     # (a trace takes weights as constants)
    cache = _cache(blk) if T == 1 else None
    with torch.no_grad():
        try:
            graph = str(torch.jit.trace(lambda x: blk(x, None, cache, 0), (x,), check_trace=False).inlined_graph)
        except AssertionError:      # (token_shift's check of the head dim refuses the tracer's sizes)
            return
    assert "aten::linear" in graph or "aten::matmul" in graph


@pytest.mark.parametrize("T", [1, 64])
def test_dispatch_modes_see_the_products_of_a_block(T):
    """A mode that counts or replaces operators gets the block's matrix products (7 projections, o_proj, two of the MLP)."""
    seen = []

    class Record(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            seen.append(func.__name__)
            return func(*args, **(kwargs or {}))

    blk, x = _block(), _x(T)
    args = (None, _cache(blk), 0) if T == 1 else ()
    with torch.no_grad(), Record():
        blk(x, *args)
    assert sum(n.split(".")[0] in ("mm", "addmm", "bmm", "matmul", "linear") for n in seen) == 10


@pytest.mark.parametrize("cls", [False, True])
@pytest.mark.parametrize("what", ["seq_start", "threshold"])
def test_arguments_changed_before_the_backward_are_noticed(what, cls):
    """The backward masks and prunes by the values of the forward, so a change in between raises."""
    q, k, v, g = _qkvg(B=2)
    q.requires_grad_()
    kw = dict(seq_start=torch.tensor([3, 9], device="cuda"), adaptive_threshold=torch.full((2, 2), -10.0, device="cuda"))
    out = (fox.ops.ForgettingAttention.apply(q, k, v, g, kw["seq_start"], True, None, kw["adaptive_threshold"]) if cls
           else fox.forgetting_attention(q, k, v, g, head_first=True, **kw))
    kw["seq_start" if what == "seq_start" else "adaptive_threshold"].add_(1)
    with pytest.raises(RuntimeError, match="inplace"):
        out.sum().backward()


def test_saved_tensor_hooks_get_all_that_attention_keeps():
    """Offloading and checkpointing work on what is saved: every array the node holds passes the hooks, and what they give
    back is used."""
    q, k, v, g = _qkvg(B=2)
    do = torch.randn(q.shape, generator=torch.Generator().manual_seed(9)).to(q.dtype).cuda()
    seq = torch.tensor([3, 9], device="cuda")
    grads, sizes = [], []
    for hooked in (False, True):
        x = [t.clone().requires_grad_() for t in (q, k, v, g)]
        pack = lambda t: (sizes.append((t.dtype, t.numel())), t.cpu())[1]
        with torch.autograd.graph.saved_tensors_hooks(*((pack, lambda t: t.cuda()) if hooked else (lambda t: t,) * 2)):
            out = fox.forgetting_attention(*x, head_first=True, seq_start=seq, adaptive_threshold=-20.0)
        out.backward(do)
        grads.append([t.grad for t in x])
    assert sum(n for d, n in sizes if d == torch.bfloat16) == 4 * q.numel()
    assert sum(n for d, n in sizes if d == torch.float32) >= 2 * g.numel()           # gate prefixes, log normalisers
    assert sum(n for d, n in sizes if d == torch.int64) == 2 + 2 * 4 * (256 // 128)   # seq_start, both index arrays
    assert torch.equal(grads[0][1], grads[1][1]) and torch.equal(grads[0][2], grads[1][2])
    for i in (0, 3):    # (sums by fp32 atomics, whose order varies: an ulp of the result's type here and there)
        a, b = [t[i].float() for t in grads]
        assert (a - b).norm() <= 2 ** -9 * b.norm()


class _Wrapped(torch.Tensor):
    """A tensor without storage of its own, as weight-only quantised weights are: every operator works on what it holds."""

    @staticmethod
    def __new__(cls, inner):
        return torch.Tensor._make_wrapper_subclass(cls, inner.size(), strides=inner.stride(), dtype=inner.dtype, device=inner.device)

    def __init__(self, inner):
        self.inner = inner

    @classmethod
    def __torch_dispatch__(cls, func, types, args=(), kwargs=None):
        unwrap = lambda t: t.inner if isinstance(t, cls) else t
        args, kwargs = torch.utils._pytree.tree_map(unwrap, (args, kwargs or {}))
        out = func(*args, **kwargs)
        return cls(out) if func is torch.ops.aten.detach.default else out


@pytest.mark.parametrize("which", ["attn.q_proj", "attn.v_proj.shift_proj", "attn.o_proj", "mlp.gate_proj", "mlp.down_proj"])
@pytest.mark.parametrize("T", [1, 64])
def test_block_with_a_weight_without_storage(which, T):
    """The module whose weight is a wrapper runs its own forward, which the subclass takes part in."""
    blk, x = _block().requires_grad_(False), _x(T)
    res = []
    for wrapped in (False, True):
        args = (None, _cache(blk), 0) if T == 1 else ()
        if wrapped:
            m = blk.get_submodule(which)
            m.weight = torch.nn.Parameter(_Wrapped(m.weight.data), requires_grad=False)
            assert type(m.weight.data_ptr()) is int and m.weight.data_ptr() == 0
        res.append(blk(x, *args).float())
    assert (res[0] - res[1]).norm() <= 2 ** -6 * res[0].norm()     # (native against modules: 8 roundings to 16 bits)


def test_attention_on_wrapped_tensors():
    """(B, T, H, D) calls permute first, which turns a wrapper of this kind into the tensor it holds."""
    args = [t.transpose(1, 2).contiguous() for t in _qkvg()]
    ref = fox.forgetting_attention(*args)
    assert torch.equal(fox.forgetting_attention(*[_Wrapped(t) for t in args]), ref)


@pytest.mark.parametrize("kind", ["log gates", "gate logits", "one row, pruned", "auto"])
def test_more_than_65535_heads_without_gradients(kind):
    """4096 sequences of 24 heads: more (b, h) than a grid's y axis has blocks."""
    q, k, v, g = _qkvg(B=4096, H=24, M=1 if kind == "one row, pruned" else 3, N=5, D=16)
    kw = dict(head_first=True, adaptive_threshold={"one row, pruned": -200.0, "auto": "auto"}.get(kind))
    with torch.no_grad():
        out = (fox.forgetting_attention_from_gate_logits if kind == "gate logits" else fox.forgetting_attention)(q, k, v, g, **kw)
    lf = torch.nn.functional.logsigmoid(g) if kind == "gate logits" else g
    for b in (0, 2730, 2731, 4095):     # (65535 = 2730 * 24 + 15)
        ref = orc.dense_forgetting_attention(*[t[b:b + 1].double().cpu() for t in (q, k, v, lf)])
        ref = ref[0] if isinstance(ref, tuple) else ref
        # five weights that sum to 1, rounded to bf16, and the result once more: 2 * 2^-9 of the largest value
        assert (out[b:b + 1].double().cpu() - ref).abs().max() <= 2 ** -8 * v[b].abs().max()


@pytest.mark.parametrize("which", ["attn_norm", "mlp_norm", "attn.output_norm", "attn.q_norm", "attn.fgate_proj"])
def test_token_step_with_vectors_that_are_not_aligned(which):
    """Norm weights and biases may be views into a flat buffer."""
    blk, x = _block(), _x(1)
    res = []
    for shifted in (False, True):
        if shifted:
            m, name = blk.get_submodule(which), "bias" if which.endswith("proj") else "weight"
            flat = torch.empty(1 + getattr(m, name).numel(), device="cuda", dtype=torch.bfloat16)
            flat[1:] = getattr(m, name).data
            setattr(m, name, torch.nn.Parameter(flat[1:]))
            assert getattr(m, name).data_ptr() % 16
        cache = _cache(blk)
        with torch.no_grad():
            res.append([blk(x, None, cache, 0)] + [t.clone() for t in cache[0]] + [cache.key_shift_cache[0].clone()])
    for a, b in zip(*res):      # (native against modules: 8 roundings to 16 bits)
        assert (a.float() - b.float()).norm() <= 2 ** -6 * a.float().norm()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_gate_bias_is_added_before_the_projection_is_rounded(dtype):
    """Projections near -40 and a bias of 40: the logits lie near 0, where a projection rounded to 16 bits on its own is wrong
    by up to half an ulp of 40 (0.125 in bf16, 0.016 in fp16).  Native and module by module each round a logit once, so the
    gates' share of the results differs by the dozen roundings of the chain."""
    C, H, T = 256, 4, 300
    blk, x, dy = _block(C, H, 512, dtype), _x(T, C, dtype), _x(T, C, dtype, seed=2)
    with torch.no_grad():
        x[..., 0] = 8.0
        h = blk.attn_norm(x)[..., 0].float()
        blk.attn.fgate_proj.weight[:, 0] = -40.0 / h.mean()
        blk.attn.fgate_proj.bias.fill_(40.0)
    res = []
    for native in (True, False):
        hook = None if native else blk.attn.q_norm.register_forward_hook(lambda *a: None)
        blk.zero_grad(set_to_none=True)
        out = blk(x)
        out.backward(dy)
        res.append([(out - x).detach(), blk.attn.fgate_proj.weight.grad[:, 1:], blk.attn.fgate_proj.bias.grad,
                    blk.attn.v_proj.linear.weight.grad])
        if hook is not None:
            hook.remove()
    tol = 12 * (2.0 ** -9 if dtype == torch.bfloat16 else 2.0 ** -12)
    for a, b in zip(*res):
        assert (a.float() - b.float()).norm() <= tol * b.float().norm()


@pytest.mark.parametrize("kernel", ["step", "sequence"])
def test_mixing_weights_are_full_fp32_sigmoids(kernel):
    """sigmoid(-87.5) = 9.98e-39 against a previous value of 1e38 makes 0.998; the approximate division gives 0 there, since
    1 + exp(87.5) lies above 2^126.  (Elsewhere it is a few fp32 ulp off, which the 16-bit result does not show.)"""
    lib, st = _lib.load(), torch.cuda.current_stream().cuda_stream
    B, H, D = 1, 2, 16
    C, ld = H * D, 4 * H * D + 8      # rows [q | k | v | ogate | fgate (H) | k mix (H) | v mix (H) | pad]
    dt = torch.bfloat16
    w = torch.ones(C, device="cuda")
    if kernel == "step":
        y = torch.zeros(B, ld, device="cuda")
        y[:, 4 * C + 2 * H:4 * C + 3 * H] = -87.5
        q, ks = torch.empty(B, C, device="cuda", dtype=dt), torch.ones(B, C, device="cuda", dtype=dt)
        vs = torch.full((B, C), 1e38, device="cuda", dtype=dt)
        k, v, g = torch.empty(B, H, 8, D, device="cuda", dtype=dt), torch.empty(B, H, 8, D, device="cuda", dtype=dt), torch.empty(B, H, 8, device="cuda")
        rc = lib.fox_step_mix(0, st, _lib.FOX_DTYPE_BF16, B, H, D, y.data_ptr(), ld, w.data_ptr(), _lib.FOX_DTYPE_FP32, w.data_ptr(),
                              _lib.FOX_DTYPE_FP32, 1e-6, None, 0, None, None, ks.data_ptr(), vs.data_ptr(), q.data_ptr(), k.data_ptr(),
                              v.data_ptr(), g.data_ptr(), 8, 0)
        got = v[:, :, 0]
    else:
        y = torch.zeros(2, ld, device="cuda", dtype=dt)
        y[:, 4 * C + 2 * H:4 * C + 3 * H] = -87.5
        y[0, 2 * C:3 * C] = 1e38
        q, k, v = torch.empty(3, 2, C, device="cuda", dtype=dt)
        rc = lib.fox_mix_fwd(0, st, _lib.FOX_DTYPE_BF16, B, 2, H, D, y.data_ptr(), ld, w.data_ptr(), w.data_ptr(), 1e-6, None,
                             q.data_ptr(), k.data_ptr(), v.data_ptr(), None, None, None)
        got = v[1]
    assert rc == 0
    ref = torch.sigmoid(torch.tensor(-87.5, dtype=torch.float64)).item() * torch.tensor(1e38).to(dt).double().item()
    assert (got.double() - ref).abs().max() <= 2 ** -8 * ref


@pytest.mark.parametrize("C,H,inter", [(256, 4, 96), (256, 2, 512), (512, 8, 1408)])
def test_long_sums_over_tokens_are_kept_in_fp32(C, H, inter):
    """Weight gradient of down_proj over 16384 tokens: the first half adds about 10^6 to every element and the second takes it
    away again.  Partial sums in fp16 overflow, whichever way the tokens are split; what is left, some thousands, does not."""
    T = 16384
    blk, x = _block(C, H, inter, torch.float16), _x(T, C, torch.float16)
    with torch.no_grad():
        blk.attn.o_proj.weight.zero_()          # the MLP's input is x itself
        x[..., 0] = 8.0
        blk.mlp.gate_proj.weight[:, 0] = 0.4
    dy = torch.where(torch.arange(T, device="cuda") < T // 2, 20.0, -20.0).half()[None, :, None].expand(1, T, C).contiguous()
    blk(x).backward(dy)
    z = x[0].double()
    m = z * torch.rsqrt(z.pow(2).mean(-1, keepdim=True) + blk.mlp_norm.eps) * blk.mlp_norm.weight.double()
    g, u = (m @ blk.mlp.gate_proj.weight.double().t()).chunk(2, -1)
    act = torch.nn.functional.silu(g) * u
    ref = dy[0].double().t() @ act
    assert (dy[0, :T // 2].double().t() @ act[:T // 2]).abs().min() > 4 * 65504 and ref.abs().max() < 65504
    # act carries about two roundings to 11 bits per token, which add up as a random walk over the tokens; the result is
    # rounded once
    walk = 20.0 * act.abs().max() * 2 * 2.0 ** -12 * T ** 0.5
    err = (blk.mlp.down_proj.weight.grad.double() - ref).abs().max()
    assert err <= 4 * walk + 2.0 ** -11 * ref.abs().max(), (err.item(), walk.item())


def test_expired_wait_after_the_last_backward_is_reported():
    """The first call after a backward usually finds its kernels still running; a record they leave later is reported by the
    calls after it, which need not be preceded by another backward, but not into a capture."""
    q, k, v, g = _qkvg()
    q.requires_grad_()
    fox.forgetting_attention(q, k, v, g, head_first=True).sum().backward()
    with torch.no_grad():
        fox.forgetting_attention(q, k, v, g, head_first=True)
        torch.cuda.synchronize()
        words = _lib.status_buffer(q.device)
        words.copy_(torch.tensor([34, 5, 96, 7], dtype=torch.int32))
        try:
            with torch.cuda.graph(torch.cuda.CUDAGraph()):
                fox.forgetting_attention(q, k, v, g, head_first=True)
            with pytest.raises(fox.FoxError, match="site=34 cta=5 thread=96 detail=7"):
                fox.forgetting_attention(q, k, v, g, head_first=True)
        finally:
            words.zero_()
        fox.forgetting_attention(q, k, v, g, head_first=True)
    fox.check_status()


@pytest.mark.parametrize("frozen", [(), ("q_proj", "v_proj.shift_proj"), ("q_proj", "k_proj", "v_proj", "ogate_proj", "fgate_proj")])
def test_block_gradients_have_memory_of_their_own(frozen):
    """A gradient that is kept or saved holds no other parameter's memory; frozen parameters get none; what is there equals
    the gradients of the block without frozen parameters."""
    blk, x, dy = _block(), _x(), _x(seed=2)
    blk(x).backward(dy)
    ref = {n: p.grad for n, p in blk.named_parameters()}
    blk.zero_grad(set_to_none=True)
    for n, p in blk.named_parameters():
        p.requires_grad_(not any(f in n for f in frozen))
    blk(x).backward(dy)
    for n, p in blk.named_parameters():
        assert (p.grad is None) == any(f in n for f in frozen)
        if p.grad is not None:
            assert p.grad.untyped_storage().nbytes() == p.numel() * p.element_size(), n
            # (sums by fp32 atomics in the attention: an ulp of the result's type here and there)
            assert (p.grad.float() - ref[n].float()).norm() <= 2 ** -8 * ref[n].float().norm(), n


@pytest.mark.parametrize("native", [True, False])
def test_pruning_threshold_is_formed_once(native, monkeypatch):
    blk, calls = _block(log_pruning_tolerance=-10.0), []
    f = fox.block.acp_threshold_from_qk_norm
    monkeypatch.setattr(fox.block, "acp_threshold_from_qk_norm", lambda *a: (calls.append(a), f(*a))[1])
    if not native:
        blk.attn.q_norm.register_forward_hook(lambda *a: None)
    out = blk(_x())
    assert len(calls) == 1 and ("FoxProBlockBackward" in out.grad_fn.name()) == native


def _peak(f):
    f()
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    f()
    torch.cuda.synchronize()
    return torch.cuda.max_memory_allocated() - before


@pytest.mark.parametrize("C,H,inter,T", [(1536, 24, 4096, 8192), (768, 12, 2048, 16384), (512, 4, 1408, 16384)])
def test_block_without_gradients_takes_no_more_memory_than_its_modules(C, H, inter, T):
    """Beside the 32 MB of the products' workspace and the stacked weights, which do not grow with the tokens, and the few
    fp32 values per head and token."""
    blk, x = _block(C, H, inter), _x(T, C)
    peak = []
    for native in (True, False):
        hook = None if native else blk.attn.q_norm.register_forward_hook(lambda *a: None)
        with torch.no_grad():
            peak.append(_peak(lambda: blk(x)))
        if hook is not None:
            hook.remove()
    fixed = (32 << 20) + 2 * (4 * C + 3 * H + 8) * C + 4 * (2 + 3 * H) * T + (1 << 20)
    assert peak[0] <= peak[1] + fixed, [p >> 20 for p in peak]


@pytest.mark.parametrize("C,H,inter", [(256, 4, 512), (512, 4, 96), (768, 12, 2048)])
@pytest.mark.parametrize("padded", [False, True])
def test_block_gives_the_same_with_and_without_gradients(C, H, inter, padded):
    """The same kernels on the same numbers, in memory that is used again without a backward: bit for bit."""
    blk, x = _block(C, H, inter), _x(700, C, B=2)
    mask = None
    if padded:
        mask = torch.ones(2, 700, dtype=torch.long, device="cuda")
        mask[0, :333] = 0
    ref = blk(x, mask)
    with torch.no_grad():
        out = blk(x, mask)
    assert ref.grad_fn is not None and out.grad_fn is None and torch.equal(out, ref)


@pytest.mark.parametrize("C,H,inter,T", [(1536, 24, 4096, 8192), (768, 12, 2048, 16384), (512, 4, 1408, 16384)])
def test_block_step_takes_little_more_memory_than_its_modules(C, H, inter, T):
    """A training step, beside the workspace of the products and the stack of weights and gradients.  The modules release
    what they saved piece by piece; the block's one node in two pieces, for which 1/16 is allowed."""
    blk, x, dy = _block(C, H, inter), _x(T, C).requires_grad_(), _x(T, C, seed=2)
    peak = []
    for native in (True, False):
        hook = None if native else blk.attn.q_norm.register_forward_hook(lambda *a: None)

        def step():
            x.grad = None
            blk.zero_grad(set_to_none=True)
            blk(x).backward(dy)

        peak.append(_peak(step))
        if hook is not None:
            hook.remove()
    fixed = (32 << 20) + 2 * 2 * (4 * C + 3 * H + 8) * C
    assert peak[0] <= peak[1] * 17 / 16 + fixed, [p >> 20 for p in peak]


def test_block_backward_twice():
    """retain_graph keeps what the first backward reads; without it a second one is refused."""
    blk, x, dy = _block(), _x(300, B=2), _x(300, B=2, seed=2)
    out = blk(x)
    out.backward(dy, retain_graph=True)
    first = {n: p.grad.clone() for n, p in blk.named_parameters()}
    blk.zero_grad(set_to_none=True)
    out.backward(dy)
    for n, p in blk.named_parameters():
        # (sums by fp32 atomics in the attention: an ulp of the result's type here and there)
        assert (p.grad.float() - first[n].float()).norm() <= 2 ** -8 * first[n].float().norm(), n
    with pytest.raises(RuntimeError, match="second time"):
        out.backward(dy)


def test_kernel_timer_times_every_launch():
    """Launches of several threads, launches by way of Python, and none that failed."""
    import threading
    q, k, v, g = _qkvg()

    def work():
        x = [t.clone().requires_grad_() for t in (q, k, v, g)]
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(20):
                fox.forgetting_attention(*x, head_first=True).sum().backward()
        torch.cuda.synchronize()

    work()
    with fox.ops.KernelTimer() as timer:
        threads = [threading.Thread(target=work) for _ in range(3)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        fox.ops.max_row_norm(k)
        fox.ops.log_lambda_cumsum(g, None)
        many = _qkvg(B=4096, H=24, M=3, N=3, D=16)
        out = fox.forgetting_attention(many[0].requires_grad_(), *many[1:], head_first=True)
        with pytest.raises(fox.FoxError, match="TOO_LARGE"):       # (the backward takes 65535 heads at most)
            out.sum().backward()
    got = timer.summary()
    assert {n: c for n, (c, _) in got.items()} == {
        "fox_attn_prologue": 61, "fox_attn_fwd": 61, "fox_bwd_delta": 60, "fox_attn_bwd": 60, "fox_bwd_finish": 60,
        "fox_max_row_norm": 1, "fox_cumsum_fwd": 1}
    assert all(0 < ms < 1e3 for _, ms in got.values())


@pytest.mark.parametrize("what", [0, 1, 2])
def test_token_step_against_a_history_with_gradients(what):
    """Frozen blocks, but keys, values or log gates in the cache that need gradients (a learned prefix): the token's output
    carries them."""
    blk, x = _block().requires_grad_(False), _x(1)
    cache, st = fox.FgateCache(), blk.attn.init_shift_state(1)
    cache.update_shift_cache(st["key_shift"], st["value_shift"], 0)
    hist = list(_qkvg(H=4, M=16, N=16)[1:])
    hist[what].requires_grad_()
    cache.update(*hist, 0)
    blk(x, None, cache, 0).sum().backward()
    assert hist[what].grad is not None and hist[what].grad.abs().sum() > 0


@pytest.mark.parametrize("eps", ["1e-6", torch.tensor(1e-6)])
@pytest.mark.parametrize("T", [1, 64])
def test_block_with_an_epsilon_that_is_no_number(eps, T):
    """A configuration may give it as text or tensor; the modules take float() of it."""
    blk, x, res = _block(), _x(T), []
    for value in (1e-6, eps):
        blk.attn_norm.eps = value
        with torch.no_grad():
            res.append(blk(x, *((None, _cache(blk), 0) if T == 1 else ())).float())
    assert (res[0] - res[1]).norm() <= 2 ** -6 * res[0].norm()     # (native against modules: 8 roundings to 16 bits)


@pytest.mark.parametrize("cls", ["FoxProAttentionLayer", "FoxMLP", "RMSNorm", "GroupNorm", "FusedGroupNormGated", "ShiftLinear", "Linear",
                                 "Module"])
@pytest.mark.parametrize("T", [1, 64])
def test_a_forward_put_on_a_class_takes_part(cls, T, monkeypatch):
    """Tools replace nn.Linear.forward, a module class's forward or nn.Module.__call__ for every instance."""
    blk, x, seen = _block(), _x(T), []
    with torch.no_grad():
        blk(x, *((None, _cache(blk), 0) if T == 1 else ()))
        owner = getattr(fox.block, cls, None) or getattr(torch.nn, cls)
        name = "__call__" if cls == "Module" else "forward"
        f = getattr(owner, name)
        monkeypatch.setattr(owner, name, lambda self, *a, **k: (seen.append(type(self)), f(self, *a, **k))[1])
        blk.forward(x, *((None, _cache(blk), 0) if T == 1 else ()))
    assert len(seen) > 0


def test_token_step_counts_as_a_change_in_place():
    """Views of the cache and shift states that were saved for a backward are seen to have been written to."""
    blk, x = _block(), _x(1)
    cache = _cache(blk)
    tensors = [*cache[0], cache.key_shift_cache[0], cache.value_shift_cache[0]]
    before = [t._version for t in tensors]
    with torch.no_grad():
        blk(x, None, cache, 0)
    assert all(t._version > v for t, v in zip(tensors, before))


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("B,T,C,H", [(2, 100, 256, 2), (1, 700, 512, 4), (2, 300, 256, 4)])
def test_block_passes_behind_one_another(B, T, C, H, graph):
    """Packing, mix, gated norm, SwiGLU, unpacking and column sums take their SMs before the kernel in front has written back.  Passes whose
    input a kernel directly in front has written, with weights changed by one between them, into memory that the allocator hands on, and a
    capture of all three: the outputs and gradients of passes that are alone, bit by bit (head dim 64, whose dQ is summed in any order: what
    depends on it to rounding)."""
    blk, base, dy = _block(C, H, 2 * C), _x(T, C, B=B), _x(T, C, seed=2, B=B)
    mask = torch.ones(B, T, dtype=torch.long, device="cuda")
    mask[0, :T // 5] = 0
    params = list(blk.parameters())
    norm = blk.mlp_norm.weight
    first = norm.detach().clone()

    def run(scale):
        with torch.no_grad():
            torch.mul(first, scale, out=norm.data)
        x = (base * scale).requires_grad_()
        out = blk(x, mask)
        return [out.detach(), *torch.autograd.grad(out, [x, *params], dy * scale)]

    scales, alone = [1.0, 0.5, 2.0], []
    for s in scales:
        torch.cuda.synchronize()
        alone.append(run(s))
        torch.cuda.synchronize()
    if graph:
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            together = [run(s) for s in scales]
        for _ in range(3):
            g.replay()
    else:
        for _ in range(4):
            together = [run(s) for s in scales]
    torch.cuda.synchronize()
    for got, want in zip(together, alone):
        assert torch.equal(got[0], want[0])
        for i, (a, b) in enumerate(zip(got[1:], want[1:])):
            if C // H == 64:
                assert (a.double() - b.double()).norm() <= 2 ** -7 * b.double().norm(), i
            else:
                assert torch.equal(a, b), i


@pytest.mark.parametrize("rows", [3, 300, 5000])
def test_norm_gate_and_swiglu_behind_one_another(rows):
    """The same for the two operators called by themselves, whose inputs a kernel directly in front has written."""
    C, H = 512, 4
    base = [_x(rows, C, seed=i)[0] for i in range(3)]
    w = torch.rand(C, device="cuda") + 0.5

    def run(scale):
        x, y, dz = [t * scale for t in base]
        x, y, wx = x.requires_grad_(), y.requires_grad_(), (w * scale).requires_grad_()
        z = fox.swiglu(fox.group_norm_gated(x, y, wx, activation="sigmoid", is_rms_norm=True, num_groups=H), y)
        return [z.detach(), *torch.autograd.grad(z, (x, y, wx), dz)]

    scales, alone = [1.0, 0.5, 2.0], []
    for s in scales:
        torch.cuda.synchronize()
        alone.append(run(s))
        torch.cuda.synchronize()
    for _ in range(4):
        together = [run(s) for s in scales]
    torch.cuda.synchronize()
    for got, want in zip(together, alone):
        for a, b in zip(got, want):
            assert torch.equal(a, b)


@pytest.mark.parametrize("rows,N", [(1, 1), (3, 4095), (4, 7168), (5, 7169), (16, 11264), (17, 11265), (148, 2000), (149, 2000), (148, 4096), (148, 4097), (149, 4097), (2, 12287), (2, 12288), (149, 12290), (2, 16383), (2, 16384), (149, 16383), (149, 16384),
                                    (150, 20000), (5, 33000)])
@pytest.mark.parametrize("dtype", ["log", torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("padded", [False, True])
def test_prefix_sums_with_and_without_loading_ahead(rows, N, dtype, padded):
    """By themselves and in a call's prologue, at the lines between the two ways: against float64, each sum to the roundings of its
    fp32 additions (4 in a thread, 10 in a block, one a chunk) and of the logarithms (4 ulp each)."""
    gen = torch.Generator(device="cuda").manual_seed(N)
    x = torch.randn(1, N, rows, generator=gen, device="cuda").transpose(1, 2) * 2 + 1     # (rows of strided gates, as a layer has them)
    x[:, :, N // 3] = -40.0
    x = x.contiguous() if rows % 2 else x
    start = 3 * N // 4 if padded else 0
    seq = torch.full((1,), start, dtype=torch.long, device="cuda") if padded else None
    if dtype == "log":
        x = torch.nn.functional.logsigmoid(x)
        lam, ref = ops.log_lambda_cumsum(x, seq), x.double()
    else:
        x = x.to(dtype)
        lam, ref = ops.gate_prefix_from_logits(x, seq), torch.nn.functional.logsigmoid(x.double())
    ref[:, :, :start] = 0
    bound = (14 + N / 4096 + 4) * 2.0 ** -23 * ref.abs().cumsum(-1)
    assert ((lam.double() - ref.cumsum(-1)).abs() <= bound).all()
    if rows * N > 4e5 or N == 1:
        return
    k = torch.randn(1, rows, N, 64, generator=gen, device="cuda").bfloat16()
    with torch.no_grad():    # (two query rows: one is a decode call, without a prologue)
        call = fox.forgetting_attention if dtype == "log" else fox.forgetting_attention_from_gate_logits
        out = call(k[:, :, -2:], k, k, x, head_first=True, seq_start=seq)[:, :, -1].double()
    s = (k.double() @ k[:, :, -1:].double().transpose(2, 3))[..., 0] / 8 + (ref.cumsum(-1)[:, :, -1:] - ref.cumsum(-1))
    s[:, :, :start] = float("-inf")
    want = (s.softmax(-1)[..., None] * k.double()).sum(2)
    assert (out - want).norm() <= 2 ** -7 * want.norm()
