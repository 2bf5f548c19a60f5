"""CPU tests of the host side: the C-ABI library loads and exports every symbol the header
declares, argument errors are reported before any launch, and the Python wrappers keep the
reference's preconditions and refuse to run without a GPU (there is no CPU fallback)."""
import ctypes
import os
import re

import pytest
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_library_exports_every_declared_symbol():
    from flashy_linear_attention_b200 import _lib

    header = open(os.path.join(ROOT, "include", "flashlinear_sm100.h")).read()
    declared = sorted(set(re.findall(r"\b(fla_sm100_\w+)\s*\(", header)))
    assert declared, "no declarations found in the header"
    lib = _lib.load()
    for name in declared:
        assert hasattr(lib, name), f"{name} is declared in include/flashlinear_sm100.h but not exported"
    assert set(declared) == set(_lib.EXPORTED_SYMBOLS)
    assert lib.fla_sm100_abi_version() == _lib.FLA_ABI_VERSION
    assert b"16" in lib.fla_sm100_strerror(-3)


def test_struct_layout_matches_header():
    # field order and count of FlaArgs in the header vs the ctypes mirror
    from flashy_linear_attention_b200._lib import FlaArgs, FlaTensor

    assert ctypes.sizeof(FlaTensor) == 32
    names = [f[0] for f in FlaArgs._fields_]
    header = open(os.path.join(ROOT, "include", "flashlinear_sm100.h")).read()
    body = header[header.index("typedef struct FlaArgs {"):header.index("} FlaArgs;")]
    body = re.sub(r"/\*.*?\*/", "", body, flags=re.S)
    decl = []
    for stmt in body.split(";"):
        stmt = stmt.replace("typedef struct FlaArgs {", "").strip()
        if not stmt:
            continue
        parts = stmt.replace("*", " ").split(",")
        first = parts[0].split()
        decl.append(first[-1])
        decl.extend(p.strip() for p in parts[1:])
    assert decl == names


def test_invalid_arguments_are_rejected_without_a_gpu():
    from flashy_linear_attention_b200 import _lib
    from flashy_linear_attention_b200._lib import FlaArgs

    lib = _lib.load()
    assert lib.fla_sm100_fwd(None) == -1
    a = FlaArgs()
    assert lib.fla_sm100_fwd(ctypes.byref(a)) == -1  # zero sizes
    assert lib.fla_sm100_bwd(ctypes.byref(a)) == -1
    a.batch, a.heads, a.seqlen, a.dk, a.dv = 1, 1, 128, 64, 64
    if not torch.cuda.is_available():
        # valid sizes but no usable device: a CUDA / device error, never a crash
        assert lib.fla_sm100_fwd(ctypes.byref(a)) in (-4, -6)
    # workspace query is pure host arithmetic
    a.batch, a.heads, a.seqlen, a.dk, a.dv, a.segments = 1, 2, 4096, 128, 128, 4
    need = lib.fla_sm100_workspace_bytes(ctypes.byref(a), 0)
    assert need >= 2 * 4 * 128 * 128 * 4
    a.segments = 1
    assert lib.fla_sm100_workspace_bytes(ctypes.byref(a), 0) == 0
    # more (batch, head) pairs than a grid dimension holds: refused before any device work
    big = FlaArgs()
    big.batch, big.heads, big.seqlen, big.dk, big.dv = 1024, 64, 128, 64, 64
    assert lib.fla_sm100_fwd(ctypes.byref(big)) == -2
    assert lib.fla_sm100_bwd(ctypes.byref(big)) == -2
    # the wide (SmallVHD) shapes never split the sequence: no scratch, one segment
    a.dk, a.dv, a.segments = 273, 64, 0
    assert lib.fla_sm100_workspace_bytes(ctypes.byref(a), 0) == 0
    assert lib.fla_sm100_workspace_bytes(ctypes.byref(a), 1) == 0
    assert lib.fla_sm100_auto_segments(ctypes.byref(a), 1) == 1
    # entry points added beside the reference's interface reject null / empty arguments as well
    z = FlaArgs()
    assert lib.fla_sm100_normalize_fwd(None, 1e-5, None) == -1
    assert lib.fla_sm100_normalize_fwd(ctypes.byref(z), 1e-5, None) == -1
    assert lib.fla_sm100_normalize_bwd_prepare(ctypes.byref(z), None, None) == -1
    assert lib.fla_sm100_normalize_bwd_sweep(ctypes.byref(z), None) == -1
    assert lib.fla_sm100_normalize_workspace_bytes(None) == 0
    assert lib.fla_sm100_pad_rows(None, None, 1, 8, 8, None) == -1
    assert lib.fla_sm100_unpad_rows(None, None, 1, 8, 8, None) == -1
    assert lib.fla_sm100_pad_rows(ctypes.c_void_p(16), ctypes.c_void_p(32), 4, 9, 12, None) == -3  # dpad % 8
    assert lib.fla_sm100_pad_rows(ctypes.c_void_p(16), ctypes.c_void_p(32), 4, 9, 8, None) == -1   # dpad < d


def test_wrappers_keep_reference_preconditions():
    from flashlinear.kernels import (
        linear_flash_wrapper_bwd,
        linear_flash_wrapper_fwd,
        linear_flash_wrapper_fwd_smallv_hd,
    )

    q = torch.zeros(1, 1, 96, 64, dtype=torch.bfloat16)
    with pytest.raises(AssertionError):  # sq % 64 != 0 (linear_attn_kernels.py:323-325)
        linear_flash_wrapper_fwd(q, q, q)
    with pytest.raises(AssertionError):
        linear_flash_wrapper_bwd(q, q, q, q)
    big = torch.zeros(1, 1, 64, 512, dtype=torch.bfloat16)
    with pytest.raises(AssertionError):  # head dim cap (linear_attn_kernels.py:322)
        linear_flash_wrapper_fwd(big, big, big)
    q = torch.zeros(1, 1, 64, 64, dtype=torch.bfloat16)
    v = torch.zeros(1, 1, 64, 24, dtype=torch.bfloat16)
    with pytest.raises(AssertionError):  # hd_v must be a power of two (smallv_hd.py:336)
        linear_flash_wrapper_fwd_smallv_hd(q, q, v)
    v = torch.zeros(1, 1, 64, 128, dtype=torch.bfloat16)
    qs = torch.zeros(1, 1, 64, 32, dtype=torch.bfloat16)
    with pytest.raises(AssertionError):  # hd_v <= hd_qk (smallv_hd.py:337)
        linear_flash_wrapper_fwd_smallv_hd(qs, qs, v)


def test_no_cpu_fallback():
    from flashlinear import LinearAttention, LinearAttentionSmallVHD

    q = torch.zeros(1, 1, 64, 64, dtype=torch.bfloat16)
    with pytest.raises(RuntimeError, match="CUDA"):
        LinearAttention.apply(q, q, q)
    v = torch.zeros(1, 1, 64, 16, dtype=torch.bfloat16)
    with pytest.raises(RuntimeError, match="CUDA"):
        LinearAttentionSmallVHD.apply(q, q, v)


def test_public_names_match_reference():
    import flashlinear
    import flashlinear.kernels as fk

    assert issubclass(flashlinear.LinearAttention, torch.autograd.Function)
    assert issubclass(flashlinear.LinearAttentionSmallVHD, torch.autograd.Function)
    for name in (
        "linear_flash_wrapper_fwd",
        "linear_flash_wrapper_bwd",
        "linear_flash_wrapper_fwd_smallv_hd",
        "linear_flash_wrapper_bwd_smallv_hd",
    ):
        assert callable(getattr(fk, name))


def test_shard_batch_heads_partitions_every_head_once():
    from flashy_linear_attention_b200.sharding import shard_batch_heads

    t = torch.arange(4 * 32).reshape(4, 32, 1, 1)
    for world in (1, 2, 4, 8, 16):
        seen = torch.cat([shard_batch_heads(t, r, world).reshape(-1) for r in range(world)])
        assert torch.equal(seen.sort().values, t.reshape(-1))
    with pytest.raises(ValueError):
        shard_batch_heads(t, 0, 3)


def test_host_pipeline_has_no_cpu_fallback():
    from flashy_linear_attention_b200.host import HostPipeline

    with pytest.raises(RuntimeError, match="CUDA"):
        HostPipeline("cpu")


@pytest.mark.parametrize("tokens", [128, 1024, 1984, 2048])
@pytest.mark.parametrize("heads", [99, 128, 296, 512, 1100])
@pytest.mark.parametrize("dim", [32, 64, 128])
def test_short_backward_never_starts_from_the_final_state(heads, tokens, dim):
    """Up to 2048 tokens dQ is summed from the start, whatever the number of heads (one late Inf would otherwise reach
    dQ of all earlier tokens): neither the single sweep nor the form with one CTA a head is taken."""
    from flashy_linear_attention_b200 import _lib

    lib = _lib.load()
    a = _lib.FlaArgs()
    a.batch, a.heads, a.seqlen, a.dk, a.dv = 1, heads, tokens, dim, dim
    assert lib.fla_sm100_bwd_uses_final_state(ctypes.byref(a)) == 0
    assert lib.fla_sm100_bwd_one_cta(ctypes.byref(a)) == 0
    assert lib.fla_sm100_normalized_bwd_workspace_bytes(ctypes.byref(a)) == 0
    a.seqlen = 2112
    assert lib.fla_sm100_bwd_uses_final_state(ctypes.byref(a)) == 1


# heads, head dim, one CTA a head, the same with the denominator's gradient inside: both sides of every line
@pytest.mark.parametrize("heads,dim,one,norm", [
    (49, 56, 0, 0), (50, 56, 1, 1), (197, 56, 1, 1), (98, 64, 0, 0), (99, 64, 1, 1), (148, 64, 1, 1), (149, 64, 0, 0), (197, 64, 0, 0),
    (198, 64, 1, 1), (98, 128, 0, 0), (99, 128, 1, 1), (148, 128, 1, 1), (149, 128, 0, 0), (197, 128, 0, 0), (198, 128, 1, 0),
    (226, 128, 1, 0), (227, 128, 1, 1), (303, 128, 0, 0), (304, 128, 1, 0), (341, 128, 1, 1), (98, 72, 0, 0), (99, 72, 1, 1),
    (197, 72, 0, 0), (198, 72, 0, 1), (226, 72, 0, 1), (227, 72, 1, 1), (340, 72, 0, 1), (341, 72, 1, 1), (198, 96, 1, 1), (303, 112, 0, 1), (304, 112, 1, 1),
    (226, 83, 0, 0), (227, 83, 1, 0), (198, 90, 1, 0)])
def test_which_heads_get_one_cta_for_their_gradients(heads, dim, one, norm):
    from flashy_linear_attention_b200 import _lib

    lib = _lib.load()
    a = _lib.FlaArgs()
    a.batch, a.heads, a.seqlen, a.dk, a.dv = 1, heads, 4096, dim, dim
    assert lib.fla_sm100_bwd_one_cta(ctypes.byref(a)) == one
    a.seqlen = 3072  # the line of 64 columns in tokens
    assert lib.fla_sm100_bwd_one_cta(ctypes.byref(a)) == (one or (dim == 64 and heads >= 50))
    assert (lib.fla_sm100_normalized_bwd_workspace_bytes(ctypes.byref(a)) > 0) == norm
    assert lib.fla_sm100_bwd_uses_final_state(ctypes.byref(a)) == 1


def test_segment_planning_queries_without_a_gpu():
    """How a call will be split is host arithmetic (148 SMs assumed when no device answers): the
    queries that size the caller's scratch must agree with each other for the shapes of the
    benchmark and its per-GPU shares."""
    from flashy_linear_attention_b200 import _lib
    from flashy_linear_attention_b200._lib import FlaArgs

    lib = _lib.load()

    def query(B, H, N, dk, dv, segments=0):
        a = FlaArgs()
        a.batch, a.heads, a.seqlen, a.dk, a.dv, a.segments = B, H, N, dk, dv, segments
        return {
            "seg_fwd": lib.fla_sm100_auto_segments(ctypes.byref(a), 0),
            "seg_bwd": lib.fla_sm100_auto_segments(ctypes.byref(a), 1),
            "ws_fwd": lib.fla_sm100_workspace_bytes(ctypes.byref(a), 0),
            "ws_bwd": lib.fla_sm100_workspace_bytes(ctypes.byref(a), 1),
            "states": lib.fla_sm100_seg_states_bytes(ctypes.byref(a)),
            "uses_final": lib.fla_sm100_bwd_uses_final_state(ctypes.byref(a)),
        }

    # the whole benchmark job: 128 heads fill the GPU, nothing is split, the backward sweeps once
    full = query(4, 32, 8192, 128, 128)
    assert full["seg_fwd"] == 1 and full["seg_bwd"] == 1
    assert full["ws_fwd"] == 0 and full["ws_bwd"] == 0 and full["states"] == 0
    assert full["uses_final"] == 1
    # its share on one of 8 GPUs: 16 heads, forward in 8 segments, backward in 3, both from one launch
    share = query(1, 16, 8192, 128, 128)
    assert share["seg_fwd"] == 8 and share["seg_bwd"] == 3
    assert share["states"] == 16 * 7 * 128 * 128 * 4      # one boundary state per segment but the first
    assert share["ws_fwd"] >= 16 * 8 * 128 * 128 * 4 and share["ws_bwd"] >= 3 * 16 * 3 * 128 * 128 * 4
    assert share["uses_final"] == 1
    # scratch states are padded to the kernel's tile: head dim 96 is sized like 128
    assert query(1, 16, 8192, 96, 96)["states"] == share["states"]
    assert query(1, 16, 8192, 64, 64)["states"] == 16 * 7 * 64 * 64 * 4
    # a long sequence whose even split (57 chunks) would not divide it gets equal segments (64)
    long = query(1, 16, 65536, 128, 128)
    assert long["states"] == 16 * 7 * 128 * 128 * 4
    # short sequences keep the two-direction backward; dk != dv and wide heads have no boundary states
    assert query(1, 16, 2048, 128, 128)["uses_final"] == 0
    assert query(1, 16, 8192, 128, 64)["states"] == 0
    assert query(1, 16, 8192, 256, 64)["states"] == 0
    # an explicit segment count is honoured
    assert query(1, 4, 8192, 128, 128, segments=4)["seg_fwd"] == 4


@pytest.mark.parametrize("heads,seqlen,dim,fwd,bwd", [
    (64, 1024, 128, 1, 1),     # two segments of a 128-wide forward never pay
    (72, 8192, 128, 1, 1),
    (48, 3072, 128, 1, 1),     # three pay from 27 chunks on
    (48, 4096, 128, 3, 1),
    (16, 1024, 128, 1, 1),     # 8 chunks: too short for any split
    (16, 2048, 128, 8, 1),     # up to 2048 tokens a split backward takes three launches
    (16, 3072, 128, 8, 3),
    (1, 2048, 128, 8, 8),
    (72, 3072, 64, 1, 1),
    (72, 8192, 64, 2, 1),
    (8, 1024, 64, 1, 1),
    (8, 2048, 64, 8, 6),
])
def test_sequences_are_split_only_where_it_pays(heads, seqlen, dim, fwd, bwd):
    from flashy_linear_attention_b200 import _lib
    from flashy_linear_attention_b200._lib import FlaArgs

    lib = _lib.load()
    a = FlaArgs()
    a.batch, a.heads, a.seqlen, a.dk, a.dv = 1, heads, seqlen, dim, dim
    got = [lib.fla_sm100_auto_segments(ctypes.byref(a), p) for p in (0, 1)]
    assert got == [fwd, bwd]
    for p, nseg in enumerate(got):  # scratch is asked for exactly where the call is split
        assert (lib.fla_sm100_workspace_bytes(ctypes.byref(a), p) > 0) == (nseg > 1)


@pytest.mark.parametrize("heads,seqlen,dk,dv,state,bwd", [
    (64, 8192, 128, 128, 2, 1),  # a state pass and the forward that reads its prefixes: 187 us whole, 168 split
    (64, 4096, 128, 128, 1, 1),  # (104 and 108)
    (56, 8192, 128, 128, 2, 1),
    (64, 1024, 64, 64, 1, 1),    # (25.0 and 25.3)
    (64, 2048, 64, 64, 2, 1),    # (40 and 33)
    (4, 1024, 128, 128, 4, 1),   # (29 and 24)
    (24, 8192, 128, 128, 6, 1),  # backward without boundary states: 117 us whole, 147 split
    (16, 4096, 128, 128, 8, 1),  # (62 and 69)
    (16, 8192, 128, 128, 8, 3),  # (114 and 109)
    (8, 3072, 128, 128, 12, 6),  # (46 and 38)
    (24, 4096, 64, 64, 6, 1),    # (43 and 48)
    (8, 2048, 128, 64, 8, 6),    # dk != dv, two calls: (57 and 54)
    (12, 2048, 128, 64, 8, 1),   # (58 and 63)
    (16, 3072, 64, 32, 8, 3),    # (65 and 55)
])
def test_split_rule_follows_what_the_call_does(heads, seqlen, dk, dv, state, bwd):
    from flashy_linear_attention_b200 import _lib
    from flashy_linear_attention_b200._lib import FLA_DEBUG_NO_FUSED_SEGMENTS, FlaArgs

    lib = _lib.load()
    a = FlaArgs()
    a.batch, a.heads, a.seqlen, a.dk, a.dv = 1, heads, seqlen, dk, dv
    assert lib.fla_sm100_auto_segments(ctypes.byref(a), 2) == state
    a.segment_states_ready = 1  # the forward that reads the prefixes must count the same segments
    assert lib.fla_sm100_auto_segments(ctypes.byref(a), 0) == state
    a.segment_states_ready = 0
    with_states = lib.fla_sm100_workspace_bytes(ctypes.byref(a), 1)
    a.debug_flags = FLA_DEBUG_NO_FUSED_SEGMENTS  # no boundary states
    assert lib.fla_sm100_auto_segments(ctypes.byref(a), 1) == bwd
    # scratch asked for with boundary states in mind covers the call that comes without
    assert with_states >= lib.fla_sm100_workspace_bytes(ctypes.byref(a), 1)


@pytest.mark.parametrize("size,strides", [((1, 1, 1, 83), (83, 83, 83, 1)), ((1, 1, 1, 64), (64, 64, 64, 1)),
                                          ((1, 3, 1, 83), (64 * 83 * 3, 64 * 83, 83, 1)), ((2, 3, 1, 20), (1920, 640, 20, 1)),
                                          ((1, 1, 1, 83), (88, 88, 88, 1)), ((1, 1, 1, 83), (84, 84, 84, 1)),
                                          ((1, 2, 64, 128), (0, 0, 128, 1)), ((1, 1, 5, 64), (8, 8, 0, 1))])
def test_addressable_is_what_the_library_accepts(size, strides):
    """A tensor that is read in place must pass the library's operand check (row stride a multiple of 8
    elements that holds the padded row, whatever the length; head and batch strides where they count)."""
    from flashy_linear_attention_b200 import ops

    t = torch.empty(64 * 83 * 3 + 512, dtype=torch.bfloat16).as_strided(size, strides)
    sb, sh, sn = strides[:3]
    accepted = sn % 8 == 0 and sn >= (size[3] + 7) // 8 * 8 and (size[1] == 1 or sh % 8 == 0) and (size[0] == 1 or sb % 8 == 0)
    assert ops._addressable(t) == accepted


def test_native_host_path_belongs_to_one_torch_and_python(monkeypatch, tmp_path):
    """The extension's file name carries both versions: after an upgrade it counts as not built (so build()
    makes it anew), and calls fall back to the ctypes path with one warning instead of an ImportError."""
    import sysconfig
    import warnings

    from flashy_linear_attention_b200 import _lib, build

    path = build.host_path()
    assert torch.__version__ in path and path.endswith(sysconfig.get_config_var("EXT_SUFFIX"))
    assert _lib.host() is not None
    monkeypatch.setattr(torch, "__version__", "99.0")
    assert build.host_path() != path and build.is_stale()
    monkeypatch.setattr(_lib, "_host", None)
    with pytest.warns(RuntimeWarning, match="flashy_linear_attention_b200.build"):
        assert _lib.host() is None
    with warnings.catch_warnings():
        warnings.simplefilter("error")
        assert _lib.host() is None  # said once
    # a file that cannot be loaded (another ABI, for one) counts the same
    bad = tmp_path / "_hostcalls.so"
    bad.write_bytes(b"not an extension")
    monkeypatch.setattr(build, "host_path", lambda: str(bad))
    monkeypatch.setattr(_lib, "_host", None)
    with pytest.warns(RuntimeWarning):
        assert _lib.host() is None


@pytest.mark.parametrize("heads, tokens, fused", [(1, 128, 1), (2, 1024, 1), (60, 1024, 1), (60, 1025, 0), (75, 4096, 0),
                                                  (76, 4096, 1), (128, 4096, 1), (2, 4096, 0)])
@pytest.mark.parametrize("width", [64, 128])
def test_rule_of_the_fused_denominator(heads, tokens, fused, width):
    """Short calls and many heads take the fused forward; a caller that asks for one segment gets it."""
    from flashy_linear_attention_b200 import _lib
    from flashy_linear_attention_b200._lib import FlaArgs

    a = FlaArgs()
    a.batch, a.heads, a.seqlen, a.dk, a.dv = 1, heads, tokens, width, width
    assert _lib.load().fla_sm100_normalized_fused(ctypes.byref(a)) == fused
    a.segments = 1
    assert _lib.load().fla_sm100_normalized_fused(ctypes.byref(a)) == 1


# 73 features: the two lines in heads and tokens, and the sizes beside them that were timed on both sides
@pytest.mark.parametrize("heads,tokens,forward,backward", [
    (1, 2048, False, False), (1, 4096, True, True), (4, 4096, True, True), (8, 4096, True, False), (8, 8192, True, True),
    (16, 3968, False, False), (16, 4096, True, False), (16, 65536, True, True), (24, 4096, False, False), (24, 8192, True, False),
    (32, 8192, False, False), (32, 16384, True, False), (40, 16384, False, False), (48, 65536, False, False), (1, 128, False, False)])
def test_raw_features_take_the_faster_way(heads, tokens, forward, backward):
    from flashy_linear_attention_b200 import ops

    assert ops._taylor_memory_is_faster(8, heads, tokens, False) == forward
    assert ops._taylor_memory_is_faster(8, heads, tokens, True) == backward
    assert not ops._taylor_memory_is_faster(16, heads, tokens, True) and not ops._taylor_memory_is_faster(16, heads, tokens, False)


def test_where_the_backward_takes_features_from_memory_the_forward_does():
    from flashy_linear_attention_b200 import ops

    for heads in range(1, 200):
        for tokens in range(64, 1 << 17, 64 * heads):
            assert ops._taylor_memory_is_faster(8, heads, tokens, False) or not ops._taylor_memory_is_faster(8, heads, tokens, True)


def test_a_call_for_the_separate_kernels_allocates_nothing(monkeypatch):
    """The denominator's gradient inside the product kernel is refused before any tensor is made (or a GPU needed)."""
    from flashy_linear_attention_b200 import ops

    q = torch.zeros(1, 16, 2176, 64, dtype=torch.bfloat16)
    s_last = torch.zeros(16, 64, 64)
    for name in ("empty", "empty_like"):
        monkeypatch.setattr(torch, name, lambda *a, **k: pytest.fail("allocated"))
    assert ops.normalized_bwd(q, None, q, q, q, s_last) is None
