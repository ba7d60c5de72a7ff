"""The C-ABI library builds, loads and exports every symbol the header declares (no GPU)."""
import ctypes
import os
import re

import pytest

from paroatten_b200 import _lib

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def declared_symbols():
    text = open(os.path.join(ROOT, "include", "paro_b200.h")).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(paro_[a-z0-9_]+)\s*\(", text)))


def test_header_symbols_exported():
    handle = _lib.lib()
    names = declared_symbols()
    assert "paro_sparse_attn" in names and len(names) >= 12
    for n in names:
        assert hasattr(handle, n), f"{n} declared in include/paro_b200.h but not exported"
    assert set(names) == set(_lib.SIGNATURES), "ctypes signatures out of sync with the header"


def test_version_and_argument_errors_without_gpu():
    handle = _lib.lib()
    assert handle.paro_version() == 100
    # argument validation happens before any CUDA call, so it can be exercised on a CPU box
    rc = handle.paro_quant_int8(None, 0, 1, 1, 64, 64, 0, 0, 64, None, 0.0, 32, None, None, None)
    assert rc == _lib.PARO_EINVAL and b"null" in handle.paro_last_error()
    buf = ctypes.create_string_buffer(64 * 96 * 2 + 64)
    addr = (ctypes.addressof(buf) + 15) & ~15
    rc = handle.paro_quant_int8(addr, 0, 1, 1, 64, 96, 0, 0, 96, None, 0.0, 32, addr, addr, None)
    assert rc == _lib.PARO_ESHAPE and b"head_dim" in handle.paro_last_error()
    rc = handle.paro_quant_int8(addr, 0, 1, 1, 64, 64, 0, 0, 64, None, 0.0, 48, addr, addr, None)
    assert rc == _lib.PARO_EINVAL and b"group" in handle.paro_last_error()
    rc = handle.paro_rope_permute(addr, addr + 16, 1, 1, 1, 10, 64, 0, 0, 64, 0, 1, 2, 3, None, 0, 0, None, None, 0, 0, None)
    assert rc == _lib.PARO_ESHAPE and b"!= N" in handle.paro_last_error()
    rc = handle.paro_plan_schedule(addr, addr, 1, 4, 70000, addr, addr, None)
    assert rc == _lib.PARO_ESHAPE and b"16 bits" in handle.paro_last_error()
    rc = handle.paro_rope_permute_norm(addr, addr + 16, 1, 1, 1, 6, 64, 0, 0, 64, 0, 1, 2, 3, None, 0, None, None, 0, 0,
                                       7, None, None, None, 1e-6, None)
    assert rc == _lib.PARO_EINVAL and b"norm_mode" in handle.paro_last_error()
    rc = handle.paro_rope_permute_norm(addr, addr + 16, 1, 1, 1, 6, 64, 0, 0, 64, 0, 1, 2, 3, None, 0, None, None, 0, 0,
                                       2, addr, None, None, 1e-6, None)
    assert rc == _lib.PARO_EINVAL and b"inv_rms" in handle.paro_last_error()
    assert handle.paro_channel_stats_scratch_bytes(1, 2, 1000, 128) == 2 * 2 * 128 * 16 + 2 * 2 * 128 * 4
    with pytest.raises(ValueError):
        _lib.check(rc)


def test_ops_refuse_cpu_tensors():
    import torch
    import paroatten_b200 as pb
    x = torch.zeros(1, 1, 64, 64, dtype=torch.float16)
    with pytest.raises(RuntimeError, match="no CPU path"):
        pb.per_warp_int8(x, x, BLKQ=64, WARPQ=32, BLKK=64)
    with pytest.raises(RuntimeError, match="no CPU path"):
        pb.compact_plan(torch.ones(1, 2, 2, dtype=torch.bool))


def aligned_buffer(size):
    buf = ctypes.create_string_buffer(size + 64)
    return buf, (ctypes.addressof(buf) + 63) & ~63


def test_pointers_that_are_read_or_written_as_vectors_must_be_aligned():
    """Refused before any CUDA call: a store of two counts, or a load of a pair's (cos, sin), at an address that is no
    multiple of its size would fault on the GPU."""
    L = _lib.lib()
    buf, a = aligned_buffer(1 << 16)
    need = L.paro_plan_scratch_bytes(1, 8, 8, 1)
    rc = L.paro_plan_offsets(a, 1, 8, 8, 1, a, a, a + 4, a, a, need, None)
    assert rc == _lib.PARO_EALIGN and b"pair_q" in L.paro_last_error()
    for cnt, kernel in ((a + 4, a), (a, a + 4)):
        rc = L.paro_plan_lists(1, 8, 8, 1, a, a, a, a, a, a, cnt, kernel, a, need, None)
        assert rc == _lib.PARO_EALIGN and b"sched_cnt" in L.paro_last_error()
    for mode, cos, sin in ((_lib.ROPE_REAL_F32, a + 4, None), (_lib.ROPE_COMPLEX_F64, a + 8, None),
                           (_lib.ROPE_COMPLEX_F64_APPROX, a + 8, a), (_lib.ROPE_COMPLEX_F64_APPROX, a, a + 8),
                           (_lib.ROPE_COMPLEX_F64_APPROX, a, None)):
        rc = L.paro_rope_permute(a, a + 4096, 1, 1, 1, 6, 64, 0, 0, 64, 0, 1, 2, 3, None, 0, mode, cos, sin, 0, 0, None)
        assert rc == _lib.PARO_EALIGN
        rc = L.paro_prep_qk_int8(a, 1, 1, 1, 6, 64, 0, 0, 64, 0, 1, 2, 3, None, mode, cos, sin, 0, 0, 32, 0, None, a, a,
                                 None, 0, None)
        assert rc == _lib.PARO_EALIGN


def test_layer_refuses_bad_arguments_before_its_first_launch():
    L = _lib.lib()
    buf, a = aligned_buffer(1 << 20)
    three = ctypes.c_int64 * 3
    st = three(128 * 64, 128 * 64, 64)
    good = dict(q=a, k=a, v=a, q_strides=st, k_strides=st, v_strides=st, dtype=_lib.BF16, B=1, H=1, N=128, D=64, n_text=8, F=2,
                Hh=3, W=20, order_ids=a, rope_mode=_lib.ROPE_COMPLEX_F64, cos_tab=a, pairs_f=10, pairs_h=11, smooth_k=1,
                smooth_v=1, plan_slices=1, out=a, out_strides=st, sm_scale=0.125, workspace=a, workspace_bytes=1 << 20)

    def refused(code, text, **changed):
        args = _lib.LayerArgs(**dict(good, **changed))
        assert L.paro_layer(args, None) == code and text in L.paro_last_error(), changed
    assert L.paro_layer(None, None) == _lib.PARO_EINVAL
    need = L.paro_layer_workspace_bytes(_lib.LayerArgs(**good))
    assert 0 < need <= 1 << 20
    assert L.paro_layer_workspace_bytes(_lib.LayerArgs(**dict(good, D=96))) == 0 and L.paro_layer_workspace_bytes(None) == 0
    refused(_lib.PARO_ESHAPE, b"sizes", N=0)
    refused(_lib.PARO_ESHAPE, b"sizes", D=96)
    refused(_lib.PARO_ECAP, b"work space", workspace_bytes=need - 1)
    refused(_lib.PARO_ECAP, b"work space", workspace=a + 8)
    refused(_lib.PARO_ECAP, b"work space", workspace=None)
    for t in "qkv":
        refused(_lib.PARO_EINVAL, t.encode() + b"): null", **{t: None})
        refused(_lib.PARO_EALIGN, t.encode() + b")", **{t: a + 2})
        refused(_lib.PARO_EALIGN, t.encode() + b")", **{t + "_strides": three(128 * 64, 128 * 64, 68)})
    refused(_lib.PARO_EINVAL, b"dtype", dtype=5)
    refused(_lib.PARO_ESHAPE, b"!= N", n_text=9)
    refused(_lib.PARO_ESHAPE, b"!= N", F=-2, n_text=248)
    refused(_lib.PARO_EINVAL, b"rope_mode", rope_mode=4)
    refused(_lib.PARO_EINVAL, b"tables missing", cos_tab=None)
    refused(_lib.PARO_ESHAPE, b"pairs_f", pairs_f=30)
    refused(_lib.PARO_EINVAL, b"norm_mode", q_norm_mode=3)
    refused(_lib.PARO_EINVAL, b"norm weight", k_norm_mode=_lib.NORM_RMS_ALL)
    refused(_lib.PARO_EINVAL, b"takes no bias", k_norm_mode=_lib.NORM_RMS_ALL, k_norm_weight=a, k_norm_bias=a)
    refused(_lib.PARO_EINVAL, b"eps", q_norm_mode=_lib.NORM_LAYER_HEAD, q_norm_weight=a, q_norm_eps=-1.0)


def test_plan_calls_refuse_bad_arguments():
    L = _lib.lib()
    buf, a = aligned_buffer(1 << 16)
    need = L.paro_plan_scratch_bytes(1, 8, 8, 1)
    assert 0 < L.paro_plan_scratch_bytes(1, 8, 8, 0) < need and L.paro_plan_scratch_bytes(0, 8, 8, 1) == 0

    def offsets(code, mask=a, slices=1, nbq=8, nbk=8, overlap=1, row_ptr=a, pair_q=a, scratch=a, size=need):
        assert L.paro_plan_offsets(mask, slices, nbq, nbk, overlap, row_ptr, a, pair_q, a, scratch, size, None) == code

    def lists(code, slices=1, nbq=8, nbk=8, overlap=1, pair_q=a, cols=a, sched=a, scratch=a, size=need):
        assert L.paro_plan_lists(slices, nbq, nbk, overlap, a, a, pair_q, cols, a, sched, a, None, scratch, size, None) == code
    for call in (offsets, lists):
        call(_lib.PARO_EINVAL, pair_q=None)
        call(_lib.PARO_ESHAPE, slices=0)
        call(_lib.PARO_ESHAPE, nbk=0)
        call(_lib.PARO_ESHAPE, nbk=0xFFFF)
        call(_lib.PARO_ESHAPE, nbq=0xFFFF, nbk=1)
        call(_lib.PARO_ESHAPE, slices=1 << 15, nbq=1 << 8, nbk=1 << 8)
        call(_lib.PARO_ECAP, size=need - 1)
        call(_lib.PARO_ECAP, scratch=None)
        call(_lib.PARO_ECAP, scratch=a + 8)
    offsets(_lib.PARO_EINVAL, mask=None)
    offsets(_lib.PARO_EINVAL, row_ptr=None)
    lists(_lib.PARO_EINVAL, cols=None)
    lists(_lib.PARO_EINVAL, sched=None)
