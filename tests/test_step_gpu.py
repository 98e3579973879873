"""Single-token kernels: the split-KV decode from the gates at the sizes where its ranges, tiles and batches end, and a
generated token through a block against the modules' own path."""
import pytest
import torch

import forgetting_transformer_b200 as fox
from forgetting_transformer_b200 import _lib
from oracle import fox_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,N,D", [(1, 2, 1, 64), (1, 1, 127, 16), (2, 3, 129, 32), (1, 1, 1025, 128), (3, 148, 1023, 64),
                                     (1, 5, 4097, 128), (1, 1, 70000, 64)])
@pytest.mark.parametrize("padded", [False, True])
def test_decode_from_gates(B, H, N, D, padded):
    """out of one query row against the dense fp32 formulation; (B, N, H) gates and permuted keys.  bf16 rounds the
    result once and takes fp32 products otherwise: every element within 2^-8 of its value and of the row's scale."""
    g = torch.Generator().manual_seed(N + D)
    q, k, v = [torch.randn(B, t, H, D, generator=g).bfloat16().cuda() for t in (1, N, N)]
    lf = torch.nn.functional.logsigmoid(torch.randn(B, N, H, generator=g) + 3).cuda()
    seq = torch.randint(0, max(1, N // 2), (B,), generator=g).cuda() if padded else None
    with torch.no_grad():
        out = fox.forgetting_attention(q, k, v, lf, seq_start=seq)
    lam = lf.double().cumsum(1)
    s = torch.einsum("bqhd,bnhd->bhn", q.double(), k.double()) / D ** 0.5 + (lam[:, -1:] - lam).transpose(1, 2)
    if padded:
        s.masked_fill_(torch.arange(N, device="cuda")[None, None, :] < seq[:, None, None], float("-inf"))
    ref = torch.einsum("bhn,bnhd->bhd", s.softmax(-1), v.double())[:, None]
    err = (out.double() - ref).abs()
    assert (err <= 2 ** -8 * ref.abs() + 2 ** -8 * ref.pow(2).mean().sqrt()).all(), err.max().item()


@pytest.mark.parametrize("splits", [1, 8, 9, 512, 513, 1024])
@pytest.mark.parametrize("N", [700, 2048])
def test_decode_takes_any_number_of_ranges(splits, N):
    """fox_attn_decode with ranges of the caller's choice, up to 1024: merged in a cluster (up to 8) or by the second kernel,
    empty ranges among them.  bf16 rounds the result once."""
    g = torch.Generator().manual_seed(N + splits)
    B, H, D = 2, 3, 64
    q, k, v = [torch.randn(B, H, t, D, generator=g).bfloat16().cuda() for t in (1, N, N)]
    lam = torch.nn.functional.logsigmoid(torch.randn(B, H, N, generator=g) + 5).cuda().cumsum(-1).contiguous()
    lib = _lib.load()
    o, L = torch.empty_like(q), torch.empty(B, H, 1, device="cuda")
    work = torch.empty(lib.fox_attn_decode_workspace_floats(B, H, D, splits), device="cuda")
    rc = lib.fox_attn_decode(0, torch.cuda.current_stream().cuda_stream, _lib.FOX_DTYPE_BF16, B, H, N, D, _lib.t4(q), _lib.t4(k),
                             _lib.t4(v), lam.data_ptr(), None, None, 0.125, _lib.t4(o), L.data_ptr(), work.data_ptr(), splits)
    assert rc == 0
    s = (q.double() @ k.double().transpose(-1, -2))[:, :, 0] / 8 + (lam[..., -1:] - lam).double()
    ref = (s.softmax(-1)[:, :, None] @ v.double())
    assert (o.double() - ref).abs().max() <= 2 ** -8 * ref.abs().max()
    assert (L[..., 0].double() - s.logsumexp(-1)).abs().max() <= 1e-5 * s.abs().max()
    assert lib.fox_attn_decode(0, None, _lib.FOX_DTYPE_BF16, B, H, N, D, _lib.t4(q), _lib.t4(k), _lib.t4(v), lam.data_ptr(), None, None,
                               0.125, _lib.t4(o), L.data_ptr(), work.data_ptr(), 1025) == -1


@pytest.mark.parametrize("B,C,H,I,N", [(1, 256, 4, 512, 1), (2, 512, 4, 1408, 130), (9, 768, 12, 2048, 64), (16, 256, 2, 96, 300)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("padded", [False, True])
def test_token_through_block_matches_modules(B, C, H, I, N, dtype, padded):
    """block_step against the same modules called one by one (a forward hook turns the native path off): three tokens;
    output, cache rows and shift states.  The module path rounds every intermediate to 16 bits: 8 roundings of relative
    size 2^-9 (bf16) or 2^-12 (fp16) in series bound the difference by about 2^-6 and 2^-9 of the scale."""
    torch.manual_seed(B + C)
    blk = fox.FoxProBlock(C, H, I, fgate_bias=2.0).cuda().to(dtype)
    with torch.no_grad():
        for m in (blk.attn_norm, blk.mlp_norm, blk.attn.q_norm, blk.attn.k_norm, blk.attn.output_norm):
            m.weight.uniform_(0.5, 1.5)
    xs = torch.randn(3, B, 1, C, device="cuda").to(dtype)
    k, v = torch.randn(2, B, H, N, C // H, device="cuda").to(dtype)
    g = torch.nn.functional.logsigmoid(torch.randn(B, H, N, device="cuda") + 3)
    mask = None
    if padded:
        mask = torch.ones(B, N + 3, dtype=torch.long, device="cuda")
        mask[0, :N // 3] = 0
    res = []
    for native in (True, False):
        cache = fox.FgateCache(granule=128)
        st = blk.attn.init_shift_state(B)
        for i, t in enumerate(st.values()):
            t.copy_(torch.linspace(-1 + i, 1, t.numel(), device="cuda").view_as(t))
        cache.update_shift_cache(st["key_shift"], st["value_shift"], 0)
        cache.update(k, v, g, 0)
        hook = None if native else blk.attn.q_norm.register_forward_hook(lambda *a: None)
        with torch.no_grad():
            outs = [blk(x, None if mask is None else mask[:, :N + 1 + i], cache, 0) for i, x in enumerate(xs)]
        if hook is not None:
            hook.remove()
        assert cache.get_seq_length() == N + 3 and cache._seen_tokens == N + 3
        res.append(outs + [t.clone() for t in cache[0]] + [st["key_shift"].clone(), st["value_shift"].clone()])
    torch.cuda.synchronize()
    _lib.check_status()
    tol = 2 ** -6 if dtype == torch.bfloat16 else 2 ** -9
    for a, b in zip(*res):
        a, b = a.float(), b.float()
        assert (a - b).abs().max() <= tol * (b.abs().max() + 1)
        assert (a - b).norm() <= tol * b.norm()


@pytest.mark.parametrize("B,T,C,H", [(1, 2, 256, 16), (2, 129, 512, 4), (3, 17, 768, 12)])
@pytest.mark.parametrize("padded", [False, True])
def test_block_native_matches_modules(B, T, C, H, padded):
    """The block as one autograd node against its modules one by one, fp16: output, input gradient and every parameter's.
    Both round intermediates to 11 bits at a dozen points: relative error of a tensor below 12 * 2^-12."""
    torch.manual_seed(T)
    blk = fox.FoxProBlock(C, H, 2 * C, fgate_bias=2.0).cuda().to(torch.float16)
    x = torch.randn(B, T, C, device="cuda").half().requires_grad_()
    dy = torch.randn(B, T, C, device="cuda").half()
    mask = None
    if padded:
        mask = torch.ones(B, T, dtype=torch.bool, device="cuda")
        mask[0, :T // 3] = False
    res = []
    for native in (True, False):
        hook = None if native else blk.attn.q_norm.register_forward_hook(lambda *a: None)
        x.grad = None
        blk.zero_grad(set_to_none=True)
        out = blk(x, mask)
        assert ("FoxProBlockBackward" in out.grad_fn.name()) == native
        out.backward(dy)
        res.append([("out", out.detach()), ("x", x.grad)] + [(n, p.grad) for n, p in blk.named_parameters()])
        if hook is not None:
            hook.remove()
    torch.cuda.synchronize()
    _lib.check_status()
    for (n, a), (_, b) in zip(*res):
        a, b = a.float(), b.float()
        assert a.shape == b.shape and (a - b).norm() <= 12 * 2 ** -12 * b.norm() + 1e-6, (n, ((a - b).norm() / b.norm()).item())


def _native_and_modules(blk, x, dy, mask=None):
    """[(name, tensor)] of the native block and of its modules one by one (a forward hook turns the native path off)."""
    res = []
    for native in (True, False):
        hook = None if native else blk.attn.q_norm.register_forward_hook(lambda *a: None)
        x.grad = None
        blk.zero_grad(set_to_none=True)
        out = blk(x, mask)
        assert ("FoxProBlockBackward" in out.grad_fn.name()) == native
        out.backward(dy)
        res.append([("out", out.detach()), ("x", x.grad)] + [(n, p.grad) for n, p in blk.named_parameters()])
        if hook is not None:
            hook.remove()
    torch.cuda.synchronize()
    _lib.check_status()
    return res


@pytest.mark.parametrize("B,T,C,H", [(1, 1100, 256, 4), (2, 1333, 512, 4), (1, 2500, 256, 16)])
@pytest.mark.parametrize("padded", [False, True])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_pruned_block_native_matches_modules(B, T, C, H, padded, dtype):
    """With log_pruning_tolerance and strong decay most key blocks are left out; head dims 64, 128 and 16, the key norms'
    bound (from 1024 keys on), ragged lengths.  A dozen roundings, and e^-10 of a row's mass that either side may prune."""
    torch.manual_seed(T)
    blk = fox.FoxProBlock(C, H, 2 * C, fgate_bias=-1.0, log_pruning_tolerance=-10.0).cuda().to(dtype)
    x = torch.randn(B, T, C, device="cuda").to(dtype).requires_grad_()
    dy = torch.randn(B, T, C, device="cuda").to(dtype)
    mask = None
    if padded:
        mask = torch.ones(B, T, dtype=torch.int32, device="cuda")
        mask[0, :T // 3] = 0
    tol = 12 * (2.0 ** -12 if dtype == torch.float16 else 2.0 ** -9) + 2 * 2.718 ** -10
    for (n, a), (_, b) in zip(*_native_and_modules(blk, x, dy, mask)):
        a, b = a.float(), b.float()
        assert a.shape == b.shape and (a - b).norm() <= tol * b.norm() + 1e-6, (n, ((a - b).norm() / b.norm()).item())


@pytest.mark.parametrize("B,T,C,H", [(1, 1200, 256, 4), (3, 1601, 256, 2), (1, 9472, 256, 4), (1, 12007, 512, 8)])
@pytest.mark.parametrize("padded", [False, True])
def test_long_block_native_matches_modules(B, T, C, H, padded):
    """Runs of 2 to 16 tokens per CTA in the token-shift kernels, and from 9472 tokens on a backward that walks several runs:
    sequences' ends inside and between runs.  Both round intermediates to 11 bits at a dozen points."""
    torch.manual_seed(T)
    blk = fox.FoxProBlock(C, H, 2 * C, fgate_bias=4.0).cuda().to(torch.float16)
    x = torch.randn(B, T, C, device="cuda").half().requires_grad_()
    dy = torch.randn(B, T, C, device="cuda").half()
    mask = None
    if padded:
        mask = torch.ones(B, T, dtype=torch.bool, device="cuda")
        mask[B - 1, :T // 3] = False
    for (n, a), (_, b) in zip(*_native_and_modules(blk, x, dy, mask)):
        a, b = a.float(), b.float()
        assert a.shape == b.shape and (a - b).norm() <= 12 * 2 ** -12 * b.norm() + 1e-6, (n, ((a - b).norm() / b.norm()).item())


@pytest.mark.parametrize("reentrant", [False, True])
def test_block_under_checkpointing(reentrant):
    from torch.utils.checkpoint import checkpoint
    torch.manual_seed(3)
    blk = fox.FoxProBlock(256, 4, 512, fgate_bias=2.0).cuda().to(torch.bfloat16)
    x = torch.randn(2, 333, 256, device="cuda").bfloat16().requires_grad_()
    dy = torch.randn(2, 333, 256, device="cuda").bfloat16()
    res = []
    for f in (blk, lambda x: checkpoint(blk, x, use_reentrant=reentrant)):
        x.grad = None
        blk.zero_grad(set_to_none=True)
        out = f(x)
        out.backward(dy)
        res.append([out.detach(), x.grad] + [p.grad for p in blk.parameters()])
    assert torch.equal(res[0][0], res[1][0])
    for a, b in zip(*res):      # (sums by fp32 atomics in the attention: an ulp of the result's type here and there)
        assert (a.float() - b.float()).norm() <= 2 ** -8 * b.float().norm()


@pytest.mark.parametrize("B,C,H,I,N", [(1, 512, 8, 1408, 2001), (3, 256, 2, 512, 1030), (1, 256, 4, 512, 6400), (16, 1536, 24, 4096, 40),
                                       (16, 512, 32, 512, 70), (2, 768, 48, 544, 129), (16, 512, 8, 512, 3100),
                                       (16, 512, 4, 512, 3100), (2, 2048, 16, 512, 5000), (1, 768, 6, 512, 4500)])
@pytest.mark.parametrize("case", ["plain", "padded", "nothing valid", "states off 16 bytes"])
def test_token_through_every_route(B, C, H, I, N, case):
    """One token by each of the step's routes: keys in 1 to 8 ranges merged by a cluster, in more or in more CTAs than a wave by
    the separate kernels, which take states that do not start on 16 bytes too; weights through shared memory and through
    registers; a sequence whose every key is padding.  Against the modules, with the tolerance of the test above (fp16)."""
    torch.manual_seed(C + N)
    blk = fox.FoxProBlock(C, H, I, fgate_bias=2.0).cuda().to(torch.float16)
    x = torch.randn(B, 1, C, device="cuda").half()
    k, v = torch.randn(2, B, H, N, C // H, device="cuda").half()
    g = torch.nn.functional.logsigmoid(torch.randn(B, H, N, device="cuda") + 3)
    mask = None
    if case in ("padded", "nothing valid"):
        mask = torch.ones(B, N + 1, dtype=torch.long, device="cuda")
        mask[0, :N // 3] = 0
        if case == "nothing valid":
            mask[B - 1] = 0
    res = []
    for native in (True, False):
        cache = fox.FgateCache(granule=128)
        st = blk.attn.init_shift_state(B)
        if case == "states off 16 bytes":
            st = {n: torch.zeros(t.numel() + 1, dtype=t.dtype, device="cuda")[1:].view_as(t) for n, t in st.items()}
        for i, t in enumerate(st.values()):
            t.copy_(torch.linspace(-1 + i, 1, t.numel(), device="cuda").view_as(t))
        cache.update_shift_cache(st["key_shift"], st["value_shift"], 0)
        cache.update(k, v, g, 0)
        hook = None if native else blk.attn.q_norm.register_forward_hook(lambda *a: None)
        with torch.no_grad():
            out = blk(x, mask, cache, 0)
        if hook is not None:
            hook.remove()
        res.append([out] + [t.clone() for t in cache[0]] + [st["key_shift"].clone(), st["value_shift"].clone()])
    torch.cuda.synchronize()
    _lib.check_status()
    for a, b in zip(*res):
        a, b = a.float(), b.float()
        assert (a - b).abs().max() <= 2 ** -9 * (b.abs().max() + 1)
        assert (a - b).norm() <= 2 ** -9 * b.norm()


@pytest.mark.parametrize("B,I", [(1, 32768), (3, 32768), (1, 24608)])
def test_token_through_a_wide_mlp(B, I):
    """Gate products whose grid of I / 8 CTAs asks for 2^32 bytes a round, and for somewhat less, of what the down product
    reads.  Against the modules, with the tolerance of the tests above (fp16)."""
    torch.manual_seed(I)
    blk = fox.FoxProBlock(256, 2, I, fgate_bias=2.0).cuda().to(torch.float16)
    x = torch.randn(B, 1, 256, device="cuda").half()
    k, v = torch.randn(2, B, 2, 70, 128, device="cuda").half()
    g = torch.nn.functional.logsigmoid(torch.randn(B, 2, 70, device="cuda") + 3)
    res = []
    for native in (True, False):
        cache = fox.FgateCache(granule=128)
        st = blk.attn.init_shift_state(B)
        cache.update_shift_cache(st["key_shift"], st["value_shift"], 0)
        cache.update(k, v, g, 0)
        hook = None if native else blk.attn.q_norm.register_forward_hook(lambda *a: None)
        with torch.no_grad():
            res.append(blk(x, None, cache, 0).float())
        if hook is not None:
            hook.remove()
    torch.cuda.synchronize()
    _lib.check_status()
    assert (res[0] - res[1]).abs().max() <= 2 ** -9 * (res[1].abs().max() + 1)
    assert (res[0] - res[1]).norm() <= 2 ** -9 * res[1].norm()


@pytest.mark.parametrize("N", [1, 130, 2001])
@pytest.mark.parametrize("route", ["one kernel", "separate kernels"])
@pytest.mark.parametrize("padded", [False, True])
def test_token_whose_gate_forgets_everything(N, route, padded):
    """Forget logits of minus infinity, of a finite value whose multiple by log2(e) overflows, and of one that leaves the older
    keys no share: the token's own value, by either route, as by the modules (bf16, eight roundings).  With a gate of NaN too:
    it acts on the older keys, where there are any."""
    torch.manual_seed(N)
    B, C, H = 2, 256, 4
    blk = fox.FoxProBlock(C, H, 512).cuda().to(torch.bfloat16)
    x = torch.randn(B, 1, C, device="cuda").bfloat16()
    k, v = torch.randn(2, B, H, N, C // H, device="cuda").bfloat16()
    g = torch.nn.functional.logsigmoid(torch.randn(B, H, N, device="cuda") + 3)
    mask = None
    if padded:
        mask = torch.ones(B, N + 1, dtype=torch.long, device="cuda")
        mask[0, :N] = 0
    for last in (2.0, float("nan")):
        with torch.no_grad():
            blk.attn.fgate_proj.bias.copy_(torch.tensor([float("-inf"), -3e38, -1e4, last]))
        res = []
        for native in (True, False):
            cache = fox.FgateCache(granule=128)
            st = blk.attn.init_shift_state(B)
            if route == "separate kernels":   # (which take states that do not start on 16 bytes)
                st = {n: torch.zeros(t.numel() + 1, dtype=t.dtype, device="cuda")[1:].view_as(t) for n, t in st.items()}
            cache.update_shift_cache(st["key_shift"], st["value_shift"], 0)
            cache.update(k, v, g, 0)
            hook = None if native else blk.attn.q_norm.register_forward_hook(lambda *a: None)
            with torch.no_grad():
                res.append(blk(x, mask, cache, 0).float())
            if hook is not None:
                hook.remove()
        assert res[1].isfinite().all() or last != last
        assert torch.equal(res[0].isfinite(), res[1].isfinite())
        a, b = res[0].nan_to_num(0, 0, 0), res[1].nan_to_num(0, 0, 0)
        assert (a - b).norm() <= 2 ** -6 * b.norm(), last


@pytest.mark.parametrize("N,D", [(2, 64), (130, 16), (1500, 128), (5000, 64), (30000, 64)])
@pytest.mark.parametrize("at", [1, 2, 5, 70, 1100])
def test_decode_from_gates_behind_one_of_minus_infinity(N, D, at):
    """The key at whose gate everything is forgotten, and those behind it, share the row; the keys before it have no weight,
    in the same range, tile and thread or in others.  Tolerance as for finite gates."""
    g = torch.Generator().manual_seed(N + at)
    at = min(at, N)
    q, k, v = [torch.randn(1, 2, t, D, generator=g).bfloat16().cuda() for t in (1, N, N)]
    lf = torch.nn.functional.logsigmoid(torch.randn(1, 2, N, generator=g) + 3).cuda()
    lf[:, 0, N - at] = float("-inf")
    with torch.no_grad():
        out = fox.forgetting_attention(q, k, v, lf, head_first=True)
    for h, n in ((0, at), (1, N)):
        lam = lf[0, h, N - n + 1:].double().flip(0).cumsum(0).flip(0)
        s = k[0, h, N - n:].double() @ q[0, h, 0].double() / D ** 0.5
        s[:-1] += lam
        ref = s.softmax(0) @ v[0, h, N - n:].double()
        err = (out[0, h, 0].double() - ref).abs()
        assert (err <= 2 ** -8 * ref.abs() + 2 ** -8 * ref.pow(2).mean().sqrt()).all(), (h, err.max().item())


@pytest.mark.parametrize("B,H,N,D,splits", [(16, 32, 513, 64, 1), (1, 592, 129, 32, 1), (2, 128, 2048, 128, 2), (10, 27, 2000, 16, 2)])
@pytest.mark.parametrize("padded", [False, True])
def test_decode_by_four_ctas_of_an_sm(B, H, N, D, splits, padded):
    """445 to 592 (b,h), one range each, and 223 to 270 in clusters of two: one wave of four CTAs to an SM in place of two or three of
    three, launched so."""
    lib = _lib.load()
    assert lib.fox_attn_decode_splits(B, H, N) == splits and lib.fox_attn_decode_per_sm(B, H, N) == 4
    test_decode_from_gates(B, H, N, D, padded)


@pytest.mark.parametrize("B,H,N,D,thr", [(1, 2, 90, 64, None), (16, 30, 700, 64, None), (1, 3, 20000, 128, None), (2, 4, 3000, 64, -4.0)])
def test_decode_calls_behind_one_another(B, H, N, D, thr):
    """A call's kernels begin behind whatever is in front: inputs written just before, results in memory that the allocator hands on.
    One range a (b,h), clusters, ranges merged by a second kernel, and a pruned call: the bits of calls that are alone."""
    gen = torch.Generator(device="cuda").manual_seed(N)
    q, k, v = (torch.randn(B, H, n, D, generator=gen, device="cuda").bfloat16() for n in (1, N, N))
    g = torch.nn.functional.logsigmoid(torch.randn(B, H, N, generator=gen, device="cuda") + 3)
    kw = {} if thr is None else dict(adaptive_threshold=thr)

    def run(scale):
        with torch.no_grad():
            return fox.forgetting_attention(q * scale, k * scale, v * scale, g * scale, head_first=True, **kw)

    scales = [1.0, 0.5, 2.0]
    alone = []
    for s in scales:
        torch.cuda.synchronize()
        alone.append(run(s))
        torch.cuda.synchronize()
    for _ in range(5):
        together = [run(s) for s in scales]
    torch.cuda.synchronize()
    for a, b in zip(together, alone):
        assert torch.equal(a, b)
