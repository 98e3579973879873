"""CPU tests of the boundary: the C-ABI library loads and exports every symbol the
header declares, and the Python host mirrors upstream's argument checks.  No compute
call is made (there is no GPU here and no CPU path in the product)."""
import ctypes
import os
import re

import pytest
import torch

import forgetting_transformer_b200 as fox
from forgetting_transformer_b200 import _lib, build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _declared_symbols():
    text = open(os.path.join(ROOT, "include", "fox_b200.h")).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(fox_[a-z0-9_]+)\s*\(", text)))


def test_header_declares_the_expected_entry_points():
    syms = _declared_symbols()
    for s in ["fox_attn_fwd", "fox_attn_bwd", "fox_cumsum_fwd", "fox_revcumsum", "fox_find_index",
              "fox_max_row_norm", "fox_bwd_delta", "fox_dq_convert", "fox_normgate_fwd", "fox_normgate_bwd",
              "fox_token_shift_fwd", "fox_token_shift_bwd", "fox_rmsnorm_fwd", "fox_rmsnorm_bwd",
              "fox_swiglu_fwd", "fox_swiglu_bwd", "fox_attn_decode", "fox_attn_bwd_dq"]:
        assert s in syms


def test_library_builds_and_exports_every_declared_symbol():
    path = build.build()
    lib = ctypes.CDLL(path)
    for s in _declared_symbols():
        assert hasattr(lib, s), f"{s} declared in include/fox_b200.h but not exported"
    lib.fox_version.restype = ctypes.c_char_p
    assert b"sm_100a" in lib.fox_version()


def test_library_exports_nothing_beyond_the_header():
    """The default build exports exactly the declared C ABI: no debug switches, no process-global hooks."""
    import subprocess
    path = build.build()
    out = subprocess.run(["nm", "-D", "--defined-only", path], capture_output=True, text=True, check=True).stdout
    exported = {line.split()[-1] for line in out.splitlines() if line.split()[-1].startswith("fox_")}
    assert exported == set(_declared_symbols()), exported ^ set(_declared_symbols())


def test_python_bindings_cover_every_declared_symbol():
    assert set(_declared_symbols()) <= set(_lib._SIGNATURES)


def test_host_extension_takes_cuda_libraries_from_pytorch():
    """No file of one CUDA installation or version is named: only PyTorch's libraries, the kernels and the C++ runtime are
    needed directly, and the extension loads with them."""
    import subprocess
    _lib.host()
    out = subprocess.run(["readelf", "-d", build.HOST_PATH], capture_output=True, text=True, check=True).stdout
    needed = re.findall(r"\(NEEDED\).*\[(.*)\]", out)
    assert "libtorch_cuda.so" in needed
    for name in needed:
        assert re.match(r"lib(torch|c10|fox_b200|stdc\+\+|gcc_s|c\b|m\b)|ld-linux", name), name


def test_host_extension_of_another_pytorch_is_not_taken(tmp_path, monkeypatch):
    """The file that is looked for holds the PyTorch version in its name: with another version installed the present one is
    neither up to date nor loaded."""
    assert torch.__version__ in os.path.basename(build.HOST_PATH) and os.path.exists(build.HOST_PATH)
    other = build.host_path("0.0.1")
    assert other != build.HOST_PATH and not os.path.exists(other)
    monkeypatch.setattr(build, "HOST_PATH", other)
    monkeypatch.setattr(_lib, "_host", None)
    monkeypatch.setenv("FOX_B200_NO_BUILD", "1")
    assert build.is_stale()
    with pytest.raises(fox.FoxError, match="cannot be loaded"):
        _lib.host()


@pytest.mark.skipif(torch.cuda.is_available(), reason="looks at the refusal alone, on addresses that hold nothing")
@pytest.mark.parametrize("dtype,per_piece", [(_lib.FOX_DTYPE_FP32, 4), (_lib.FOX_DTYPE_BF16, 8)])
def test_cross_entropy_refuses_rows_of_too_many_pieces(dtype, per_piece):
    """A thread counts a row's 16-byte pieces in 32 bits and steps past its end: rows of more than 2^30 pieces are refused
    before anything is launched (there is no device here: smaller ones get as far as FOX_ERR_DEVICE)."""
    lib = _lib.load()
    for cols, rc in (((2 ** 30 + 1) * per_piece, -8), (2 ** 20 * per_piece, -7)):
        f = lib.fox_cross_entropy_fwd(0, None, dtype, 1, cols, 4096, cols, 4096, 0.0, 1.0, 0.0, -100, 4096, 4096, 4096)
        b = lib.fox_cross_entropy_bwd(0, None, dtype, 1, cols, 4096, cols, 4096, 4096, 4096, 1, 0.0, 1.0, 0.0, -100, 4096, cols)
        assert (f, b) == (rc, rc)


def _inputs(B=1, H=2, M=8, N=8, D=64, dtype=torch.bfloat16):
    q = torch.zeros(B, H, M, D, dtype=dtype)
    k = torch.zeros(B, H, N, D, dtype=dtype)
    v = torch.zeros(B, H, N, D, dtype=dtype)
    lf = torch.zeros(B, H, N, dtype=torch.float32)
    return q, k, v, lf


def test_dtype_assertions_match_upstream():
    q, k, v, lf = _inputs(dtype=torch.float32)
    with pytest.raises(AssertionError, match="Only torch.float16 or torch.bfloat16"):
        fox.forgetting_attention(q, k, v, lf, head_first=True)
    q, k, v, lf = _inputs()
    with pytest.raises(AssertionError, match="log_fgate must be in torch.float32"):
        fox.forgetting_attention(q, k, v, lf.half(), head_first=True)


def test_shape_assertions_match_upstream():
    q, k, v, lf = _inputs(D=48)
    with pytest.raises(AssertionError, match="head dims in"):
        fox.forgetting_attention(q, k, v, lf, head_first=True)
    q, k, v, lf = _inputs(M=16, N=8)
    with pytest.raises(AssertionError, match="longer than the query"):
        fox.forgetting_attention(q, k, v, lf, head_first=True)
    q, k, v, lf = _inputs()
    with pytest.raises(AssertionError):
        fox.forgetting_attention(q, k, v, lf[:, :1], head_first=True)
    with pytest.raises(AssertionError, match="groupped query attention"):
        fox.forgetting_attention(q, k[:, :1], v[:, :1], lf, head_first=True)


def test_no_cpu_fallback():
    q, k, v, lf = _inputs()
    with pytest.raises(_lib.FoxError, match="no CPU path"):
        fox.forgetting_attention(q, k, v, lf, head_first=True)
    with pytest.raises(_lib.FoxError, match="no CPU path"):
        fox.group_norm_gated(torch.zeros(2, 128, dtype=torch.bfloat16), torch.zeros(2, 128, dtype=torch.bfloat16),
                             torch.ones(128), is_rms_norm=True, activation="sigmoid", num_groups=2)


def test_norm_gate_rejects_unbuilt_configurations():
    x = torch.zeros(2, 128, dtype=torch.bfloat16)
    with pytest.raises(NotImplementedError):
        fox.group_norm_gated(x, x, torch.ones(128), activation="swish", is_rms_norm=True, num_groups=2)
    with pytest.raises(NotImplementedError):
        fox.group_norm_gated(x, x, torch.ones(128), activation="sigmoid", is_rms_norm=False, num_groups=2)
    with pytest.raises(ValueError):
        fox.FusedGroupNormGated(3, 128)
    m = fox.FusedGroupNormGated(2, 128, is_rms_norm=True, eps=1e-6, activation="sigmoid")
    assert torch.all(m.weight == 1) and m.bias is None


def test_tma_ready_predicate():
    x = torch.zeros(2, 16, 4, 64, dtype=torch.bfloat16)
    assert _lib.tma_ready(x) and _lib.tma_ready(x.permute(0, 2, 1, 3))
    assert not _lib.tma_ready(x[..., 1:])            # base off by 2 bytes
    assert not _lib.tma_ready(x.transpose(2, 3))     # inner stride != 1
    y = torch.zeros(2, 16, 4, 68, dtype=torch.bfloat16)[..., :64]
    assert not _lib.tma_ready(y)                     # 136-byte row stride


def test_signature_matches_upstream():
    import inspect
    sig = inspect.signature(fox.forgetting_attention)
    names = list(sig.parameters)
    assert names == ["q", "k", "v", "log_fgate", "head_first", "seq_start", "sm_scale", "adaptive_threshold"]
    for n in names[4:]:
        assert sig.parameters[n].kind is inspect.Parameter.KEYWORD_ONLY
    assert sig.parameters["head_first"].default is False
    assert sig.parameters["seq_start"].default is None


def test_layer_glue_expressions():
    """The layer-side helpers restate upstream's expressions (modeling_forgetting_transformer.py:371-396)."""
    import math
    import forgetting_transformer_b200 as fox
    mask = torch.tensor([[0, 0, 1, 1, 1], [1, 1, 1, 1, 1]])
    assert fox.seq_start_from_attention_mask(mask).tolist() == [2, 0]
    g = torch.Generator().manual_seed(0)
    H, D, T, tol = 3, 64, 1000, -10.0
    wq, wk = torch.randn(H * D, generator=g), torch.randn(H * D, generator=g)
    thr = fox.acp_threshold_from_qk_norm(wq, wk, H, D, T, tol)
    ref = -(2 * wq.view(H, D).abs().max(-1).values * wk.view(H, D).abs().max(-1).values * math.sqrt(D)
            + math.log(T)) + tol
    assert thr.shape == (H,) and torch.equal(thr, ref)
    ws = fox.acp_threshold_from_qk_norm(wq[:D], wk[:D], H, D, T, tol, share_param_across_head=True)
    assert ws.dim() == 0 and ws.item() == (-(2 * wq[:D].abs().max() * wk[:D].abs().max() * math.sqrt(D)
                                              + math.log(T)) + tol).item()


@pytest.mark.parametrize("bh", [1, 24, 49, 50, 72, 144, 223, 256, 270, 271, 400, 401, 444, 445, 512, 540, 541, 592, 593, 889, 65535])
@pytest.mark.parametrize("n", [1, 256, 257, 1279, 1500, 2000, 4099, 70000, 2 ** 31 - 2048])
def test_decode_ranges_fill_whole_waves(bh, n):
    """Ranges of one-token attention: at least 128 keys each, and never more CTAs than the waves they are cut for hold: 444 a wave, 400
    where clusters merge, or 592 and 540 where they come four to an SM.  Those are chosen only where more (b,h) than one range of a
    wave of three holds make them few, and the waves do not become more."""
    lib = _lib.load()
    s, per = lib.fox_attn_decode_splits(1, bh, n), lib.fox_attn_decode_per_sm(1, bh, n)
    assert 1 <= s <= min(512, max(1, -(-n // 128))) and per in (3, 4)
    full, clustered = (444, 400) if per == 3 else (592, 540)
    waves = -(-bh // full) + (1 if -(-bh // full) * clustered // bh <= 1 else 0)
    assert s == 1 or bh * s <= waves * (full if s > 8 else clustered)
    if per == 4:
        assert bh > 222 and -(-bh * s // (clustered if 1 < s <= 8 else full)) <= -(-bh // 444) + 1
    if bh in (270, 592) and n in (1500, 2000, 4099):
        assert (s, per) == ({270: 2, 592: 1}[bh], 4)


@pytest.mark.parametrize("grid", [1, 176, 2048, 4095, 4096, 4097, 8192, 12288, 2 ** 20])
def test_requests_ahead_of_a_token_product_cover_the_array_once(grid):
    """fox_step_product_ahead's threads ask for one 4096-byte piece after another of what a later product reads: blocks follow
    one another, then threads, then rounds, without a gap, a repetition or a round of no length, at grids beyond 2^32 bytes a
    round (4096 CTAs of 256 threads) too."""
    at = _lib.load().fox_step_ahead_offset
    assert at(grid, 0, 0, 0) == 0
    for k in (0, 1, 5):
        for thread in range(256):
            for block in {0, 1, grid // 2, grid - 2} & set(range(grid - 1)):
                assert at(grid, block + 1, thread, k) == at(grid, block, thread, k) + 4096
            after = at(grid, 0, thread + 1, k) if thread < 255 else at(grid, 0, 0, k + 1)
            assert after == at(grid, grid - 1, thread, k) + 4096


def _device_functions(text):
    """name -> parameters and body of every __global__ and __device__ function of a source without comments."""
    found = {}
    for start in re.finditer(r"__(?:global|device)__", text):
        name = re.compile(r"(\w+)\s*\(").search(text, start.end())
        while name and name.group(1) == "__launch_bounds__":
            name = re.compile(r"(\w+)\s*\(").search(text, text.index(")", name.end()))
        if not name or ";" in text[start.end():name.start()]:
            continue
        at, depth = name.end(), 1
        while depth:
            depth += {"(": 1, ")": -1}.get(text[at], 0)
            at += 1
        if not text[at:].lstrip().startswith("{"):
            continue
        at = text.index("{", at) + 1
        depth = 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[at], 0)
            at += 1
        found[name.group(1)] = found.get(name.group(1), "") + text[name.start():at]
    return found


def _sources():
    strip = lambda name: re.sub(r"//[^\n]*", "", open(os.path.join(build.CSRC, name)).read())
    common = _device_functions(strip("fox_common.cuh"))
    for name in build.SOURCES:
        yield name, strip(name), common


def _with_all_it_calls(kernel, functions):
    """The kernel, the functions that it names, those that they name, and so on."""
    reached, todo = {}, [kernel]
    while todo:
        name = todo.pop()
        reached[name] = functions[name]
        todo += [f for f in set(re.findall(r"\w+", functions[name])) & set(functions) if f not in reached and f not in todo]
    return reached


WAITS = ("griddepcontrol.wait", "pdl_wait()", "wait_for_kernel_in_front()")


def test_kernels_that_begin_early_take_no_invariant_pointers():
    """A kernel with griddepcontrol.wait may begin before the kernel in front has written what it reads: a load through a
    `const __restrict__` pointer, by __ldg or on the read-only path (.nc) is one that may be done in front of the wait.  None in
    such a kernel, nor in any function that it reaches, but for a token product's weights, which no kernel writes."""
    waiting, helpers = set(), set()
    for name, text, common in _sources():
        functions = {**common, **_device_functions(text)}
        for kernel in functions:
            if not re.search(r"__global__[^;{]*\b%s\s*\(" % kernel, text) or not any(w in functions[kernel] for w in WAITS):
                continue
            waiting.add(kernel)
            for f, body in _with_all_it_calls(kernel, functions).items():
                helpers.add(f)
                assert not any(x in body for x in ("__restrict__", "__ldg", ".nc.")) or f == "ldg_stream", (name, kernel, f)
    assert len(waiting) >= 22
    # the walk sees helpers of the common header, of two template arguments, and those that only helpers call
    assert {"ld_f32_here", "dec_store", "load_gate", "norm_part", "tma_load_4d"} <= helpers and "ldg_v4_here" not in helpers


def test_kernels_launched_behind_another_wait_for_it():
    """Each kernel that a host function gives to launch_behind(), or to cudaLaunchKernelEx with its attributes, waits in its own body."""
    launched = set()
    for name, text, _ in _sources():
        functions = _device_functions(text)
        for host in text.split("\n}\n"):
            if "launch_behind(" in host or "cudaLaunchKernelEx(" in host:
                assert "<<<" not in host, name     # (or the names below would not all be launched so)
                kernels = set(re.findall(r"\bfox_\w+_kernel\b", host))
                assert kernels, (name, host[-200:])
                for k in kernels:
                    assert any(w in functions[k] for w in WAITS), (name, k)
                launched |= kernels
    assert {"fox_attn_fwd_kernel", "fox_attn_bwd_kernel", "fox_attn_bwd_kv_kernel", "fox_attn_bwd_dq2_kernel", "fox_find_index_kernel",
            "fox_prologue_kernel", "fox_delta_kernel", "fox_bwd_finish_kernel", "fox_mix_fwd_kernel", "fox_mix_bwd_kernel", "fox_pack_kernel",
            "fox_unpack_kernel", "fox_column_sums_kernel", "fox_swiglu_fwd_kernel", "fox_swiglu_bwd_kernel", "fox_normgate_fwd_kernel",
            "fox_normgate_bwd_kernel", "fox_decode_kernel", "fox_decode_merge_kernel", "fox_step_product_kernel", "fox_step_mix_kernel",
            "fox_ce_mean_kernel"} <= launched


@pytest.mark.parametrize("units,tiles", [(1, 1), (1, 148), (37, 4), (148, 1), (74, 2), (49, 3), (1, 149), (37, 5), (150, 1), (28, 65), (65535, 7),
                                         (100000, 1), (3, 70000), (2 ** 31 - 70000, 1), (2 ** 31 + 5, 1), (2 ** 32 - 131071, 1)])
@pytest.mark.parametrize("mb", [0.001, 1.9, 5, 24, 25, 60])
def test_groups_of_items_by_length(units, tiles, mb):
    """Units that go by length together: all of them where every tile has an SM to itself, so that no CTA without an item takes a
    place there; else as many as stay in 48 MB, in groups that differ by less than their number, at most 65535 of them, whose
    padded size stays below 2^31.  Units that an int does not count go one by one."""
    group = _lib.load().fox_attn_item_group(units, tiles, int(mb * 2 ** 20))
    assert 1 <= group <= units
    if units * tiles <= 148:
        assert group == units
    elif group > 1:
        groups = -(-units // group)
        assert group * mb * 2 ** 20 <= 48 * 2 ** 20 + group and groups <= 65535 and tiles <= 65535
        assert groups * group - units < group and groups * group < 2 ** 31
    if units > 2 ** 31 - 65536:
        assert group == 1


def test_scan_kernels_leave_room_for_a_second_block(tmp_path):
    """Blocks of 1024 threads: 32 registers a thread let two be on an SM.  Prologue, backward's end, and the prefix sums that do not load
    ahead (which those that do give up knowingly)."""
    import subprocess
    out = subprocess.run([os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc"), "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17",
                          "-Xptxas", "-v", "-c", os.path.join(build.CSRC, "fox_scan.cu"), "-o", str(tmp_path / "scan.o")],
                         capture_output=True, text=True, check=True).stderr
    used = dict(re.findall(r"Compiling entry function '(\w+)'.*?Used (\d+) registers", out, re.S))
    two = {k: int(r) for k, r in used.items() if re.search(r"fox_(prologue|bwd_finish)_kernel|fox_cumsum_kernelILi\dELb0E", k)}
    assert len(two) == 28 + 8 + 4 and all(r <= 32 for r in two.values()), two


@pytest.mark.parametrize("bh", [1, 9, 10, 24, 35, 48, 60, 64, 70, 71, 96, 98, 99, 140, 147, 148, 149, 296, 297, 4000])
@pytest.mark.parametrize("n,d", [(1024, 64), (4096, 128), (8192, 128), (16384, 64), (1024, 16), (12300, 16), (2 ** 24, 128)])
def test_key_norm_parts_fill_a_wave_and_stay_short(bh, n, d):
    """Key-norm parts beside the prefix scans: as fox_norm_parts, or one less where that makes one wave of 296 blocks, at least
    280 of them, and no part becomes more than half as long again; long rows of many (b,h) keep three,
    long ones of 16 or 32 channels all."""
    lib = _lib.load()
    parts, most = lib.fox_key_norm_parts(1, bh, n, d), lib.fox_norm_parts(1, bh, n, d)
    assert 1 <= parts <= most <= 32 and (parts == most or most - parts <= max(1, most // 3))
    if parts < most:
        assert 280 <= (1 + parts) * bh <= 296 and parts >= 2 and (n <= 4096 or d >= 64 and (parts >= 3 or d == 64))
    assert bh not in (70, 140, 147, 148) or parts == most


def test_sizes_for_calls_without_batch_or_heads():
    """What the C interface says about launches for no (b,h) at all is an answer, not a division by zero."""
    lib = _lib.load()
    for b, h in ((0, 4), (4, 0), (0, 0)):
        assert lib.fox_attn_decode_splits(b, h, 100) == 1 and lib.fox_step_attn_splits(b, h, 100) == 0
        assert lib.fox_norm_parts(b, h, 2048, 64) == lib.fox_key_norm_parts(b, h, 2048, 64) == 1
