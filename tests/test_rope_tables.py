"""The fp32 copy of an fp64 angle table is that of the table as it is when the passes read it."""
import ctypes

import pytest
import torch

import paroatten_b200 as pb
from oracle import paro_oracle as po
from paroatten_b200 import _lib

DEV = "cuda"


@pytest.mark.parametrize("inference", [False, True])
def test_copy_handed_to_a_pass_is_that_of_the_table(inference):
    """However the table was written to: in place (inference mode counts no versions), through .data, through an alias."""
    with torch.inference_mode(inference):
        r = pb.rope_tables((2, 3, 4), 64, "wan", device="cpu")
    writes = [lambda: r.cos.fill_(0.25), lambda: r.cos.data.fill_(0.5), lambda: r.cos.data.numpy().fill(0.75)]
    for write in writes:
        before = r.call_args()
        with torch.inference_mode(inference):
            write()
        args = r.call_args()
        assert args[0] == _lib.ROPE_COMPLEX_F64_APPROX and args[1] == r.cos.data_ptr()
        copy = (ctypes.c_float * r.cos.numel()).from_address(args[2])
        assert list(copy) == r.cos.flatten().tolist()
        del before


def separate(r):
    """The same angles as two tables, which no pass takes a copy of."""
    s = pb.RopeTables(r.mode, r.cos[..., 0], r.cos[..., 1], r.pairs_f, r.pairs_h)
    s.cos, s.sin = r.cos[..., 0].contiguous(), r.cos[..., 1].contiguous()
    return s


@pytest.mark.gpu
@pytest.mark.parametrize("how", ["inference", "data", "alias", "stream"])
def test_rewritten_table_is_followed(how):
    """Sizes at which the passes and the layer use the copy; the bits of the passes on separate tables."""
    grid, D, H = (4, 40, 52), 128, 16
    N = grid[0] * grid[1] * grid[2]
    x = torch.randn(1, H, N, D, device=DEV, generator=torch.Generator(DEV).manual_seed(1)).to(torch.bfloat16)
    assert x.numel() >= pb.rope.FP32_COPY_ELEMS
    ids = torch.arange(H, dtype=torch.int32, device=DEV) % 6
    plan = pb.compact_plan(po.make_mask(H, (N + 63) // 64, 0.3, seed=1).to(DEV))
    with torch.inference_mode(how == "inference"):
        r = pb.rope_tables(grid, D, "wan")
    layer = lambda rope: pb.paro_attention(x, x, x, ids, plan, grid_fhw=grid, rope=rope)
    layer(r), pb.rope_permute(x, ids, grid, 0, r)
    new = pb.rope_tables(grid, D, "wan", theta=50.0).cos
    if how == "inference":
        with torch.inference_mode():
            r.cos.copy_(new)
    elif how == "data":
        r.cos.data.copy_(new)
    elif how == "alias":
        torch.from_dlpack(r.cos.detach()).copy_(new)
    stream = torch.cuda.current_stream()
    if how == "stream":      # the first pass after the write is on another stream than the second
        r.cos.copy_(new)
        done = stream.record_event()
        other = torch.cuda.Stream()
        other.wait_event(done)
        with torch.cuda.stream(other):
            first = pb.rope_permute(x, ids, grid, 0, r)
        first.record_stream(stream)
    got, rows = layer(r), pb.rope_permute(x, ids, grid, 0, r)
    s = separate(r)
    torch.cuda.synchronize()
    assert torch.equal(rows, pb.rope_permute(x, ids, grid, 0, s)) and torch.equal(got, layer(s))
    q8, qs, _ = pb.prep_qk_int8(x, ids, grid, 0, r, group=32)
    w8, ws, _ = pb.prep_qk_int8(x, ids, grid, 0, s, group=32)
    assert torch.equal(q8, w8) and torch.equal(qs, ws)


@pytest.mark.gpu
def test_captured_layer_follows_the_table():
    """A replayed graph reads what the table holds at the replay."""
    grid, D, H = (4, 40, 52), 128, 4
    N = grid[0] * grid[1] * grid[2]
    x = torch.randn(1, H, N, D, device=DEV, generator=torch.Generator(DEV).manual_seed(2)).to(torch.bfloat16)
    plan = pb.compact_plan(po.make_mask(H, (N + 63) // 64, 0.3, seed=1).to(DEV))
    pplan = pb.PermutePlan({"permute": torch.tensor([[0, 3, 1, 5]])}, grid)
    r = pb.rope_tables(grid, D, "wan")
    layer = lambda rope: pb.paro_attention(x, x, x, pplan, plan, grid_fhw=grid, rope=rope)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        layer(r)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        out = layer(r)
    r.cos.copy_(pb.rope_tables(grid, D, "wan", theta=50.0).cos)
    graph.replay()
    torch.cuda.synchronize()
    got = out.clone()
    del graph
    assert torch.equal(got, layer(separate(r)))


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("scale", [1.0, 300.0, 1e35, 1e300, 1e-38, 1e-44, 1e-300])
def test_fp32_shortcut_at_the_ends_of_the_ranges(dtype, scale):
    """The fp64 rotation with the fp32 copy against the one without, bit for bit: every pair of zeros, subnormals, values at
    the end of the range, Inf and NaN, on tables up to and past the ends of fp32's range."""
    fi = torch.finfo(dtype)
    special = [0.0, -0.0, fi.smallest_normal / 4, -fi.smallest_normal, 1.0, -1.5, 1e4, -fi.max, fi.max, float("inf"),
               float("-inf"), float("nan")]
    pair = torch.tensor([[a, b] for a in special for b in special]).to(dtype)         # [144, 2]
    D, H = 64, 2
    N = pair.shape[0] * 6
    x = pair.repeat(6, 1).unsqueeze(1).expand(N, D // 2, 2).reshape(1, 1, N, D).expand(1, H, N, D).contiguous().to(DEV)
    g = torch.Generator().manual_seed(3)
    ang = torch.rand(1 + 1 + N, D // 2, dtype=torch.float64, generator=g) * 7
    tab = torch.stack([ang.cos(), ang.sin()], dim=-1).mul(scale).to(DEV)
    copy = tab.to(torch.float32)
    outs = []
    for mode, sin in ((_lib.ROPE_COMPLEX_F64, None), (_lib.ROPE_COMPLEX_F64_APPROX, copy)):
        out = torch.empty(1, H, N, D, dtype=dtype, device=DEV)
        _lib.check(_lib.lib().paro_rope_permute(
            x.data_ptr(), out.data_ptr(), _lib.dtype_code(dtype), 1, H, N, D, x.stride(0), x.stride(1), x.stride(2), 0, 1, 1, N,
            None, 0, mode, tab.data_ptr(), _lib.ptr(sin), 0, 0, _lib.stream_ptr()))
        outs.append(out.view(torch.int16))
    assert torch.equal(*outs)
