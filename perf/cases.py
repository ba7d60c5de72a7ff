"""The work that users of this package have it do, as timed cases.

    listed()            the cases, by name
    draw(rng)           one more case of the same ranges
    prepare(case, seed) what a program holds before the call: activations, plan, tables, handle
    run(state)          one pass through the public entry points
    work(case)          bytes and operations that the pass cannot do without
    tolerance(case)     how far another correct implementation of the same precision may be off

Kinds of case:

    attention  paro_attention: one self-attention layer from natural-order Q, K, V to natural-order O
    operator   paroattn_qk_int8_pv_fp16_cuda: the drop-in operator on reordered Q, K, V with a boolean block mask
    prep       the pre-attention pipeline alone: RoPE + reorder + INT8 Q, smoothed INT8 K, FP8 V
    plan       compact_plan of one (timestep bin, layer) slice of a block mask
    merge      merge_attention_states of two partial results
    host       HostPipelinedAttention: activations in pinned host memory

Activations are N(0,1) with a per-channel K offset of N(0,2), rounded to the case's data type; head orders are uniform over
the six F/H/W orders; block masks are Bernoulli with the diagonal, a local band and the text rows and columns kept.
"""
import math

import torch

import paroatten_b200 as pb

BLOCK = 64
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}

# a case's options and what they are when it does not name them
DEFAULTS = dict(B=1, n_text=0, dtype="bf16", layout="HND", family="wan", norm="none", density=0.3, window=0, lse=False)


def _case(name, kind, **kw):
    return dict(DEFAULTS, name=name, kind=kind, **kw)


def listed():
    return [
        # Wan2.1-14B, 720p: one layer on one GPU, the largest call there is
        _case("wan14b_720p", "attention", H=40, D=128, F=21, Y=45, X=80, density=0.2),
        # the same layer with its heads split over eight GPUs: what each of them runs
        _case("wan14b_720p_5_heads", "attention", H=5, D=128, F=21, Y=45, X=80, density=0.2),
        # Wan2.1-1.3B, 480p with classifier-free guidance, as its processor calls it: [B,N,H,D] projections, RMS norm of Q and K
        _case("wan1p3b_480p", "attention", B=2, H=12, D=128, F=21, Y=30, X=52, density=0.3, window=1, layout="NHD",
              norm="rms"),
        # CogVideoX-5b with guidance, as its processor calls it: joint text + video sequence, LayerNorm of Q and K
        _case("cogvideox_5b", "attention", B=2, H=48, D=64, F=13, Y=30, X=45, n_text=226, density=0.3, layout="NHD",
              family="cogvideox", norm="layer"),
        # a preview-sized call, 1024 tokens and two heads: launches and host time are what it costs
        _case("small_fp16", "attention", H=2, D=64, F=4, Y=16, X=16, dtype="fp16", family="none", density=0.5),
        # a mid-sized call with nothing even about it: odd grid, text tokens, ragged last block, LSE wanted by a ring step
        _case("ragged_lse_fp16", "attention", H=6, D=128, F=3, Y=37, X=53, n_text=77, dtype="fp16", density=0.4, window=2,
              lse=True),
        # the reference's operator as its processors call it: reordered tensors, the layer's boolean mask handed over per call
        _case("operator_mask_fp16", "operator", H=12, D=128, F=21, Y=30, X=52, dtype="fp16", density=0.3, window=1),
        # the pre-attention pipeline alone on the CogVideoX-5b shape
        _case("prep_cogvideox_5b", "prep", B=2, H=48, D=64, F=13, Y=30, X=45, n_text=226, family="cogvideox"),
        # first use of a (timestep bin, layer) slice of the Wan2.1-14B plan; a video needs hundreds of them
        _case("plan_wan14b_720p", "plan", H=40, D=128, F=21, Y=45, X=80, density=0.2),
        # combining the partial results of two ring steps
        _case("merge_wan1p3b_480p", "merge", H=12, D=128, F=21, Y=30, X=52),
        # activations offloaded to host memory, copied in and out by head groups
        _case("host_wan1p3b_480p", "host", H=12, D=128, F=21, Y=30, X=52, density=0.3, window=1),
    ]


# limits of a drawn case: the largest listed one
_MAX_ELEMS = 40 * 75600 * 128
_MAX_WALK = 40 * 1182 * 1182 * 0.2 * 128
_MAX_MASK = 40 * 1182 * 1182


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_grid(rng, lo, hi):
    n = _log_uniform(rng, lo, hi)
    F = min(rng.randint(1, 21), max(1, n // 16))
    yx = max(1, n // F)
    Y = max(1, min(yx, int(round(math.sqrt(yx * rng.uniform(0.4, 1.0))))))
    return F, Y, max(1, yx // Y)


def draw(rng):
    kind = rng.choices(["attention", "operator", "prep", "plan", "merge", "host"], [12, 3, 3, 2, 2, 1])[0]
    while True:
        D = rng.choice([64, 128, 128])
        family = ("cogvideox" if D == 64 else "wan") if rng.random() < 0.8 else rng.choice(["cogvideox", "wan", "none"])
        F, Y, X = _draw_grid(rng, 256, 75600)
        c = dict(DEFAULTS, kind=kind, B=rng.choice([1, 1, 2]), H=_log_uniform(rng, 1, 48), D=D, F=F, Y=Y, X=X,
                 n_text=rng.choice([0, rng.randint(1, 256), 226]) if family == "cogvideox" else 0,
                 dtype=rng.choice(["bf16", "bf16", "fp16"]), layout=rng.choice(["HND", "NHD"]), family=family,
                 density=round(rng.uniform(0.15, 0.5), 3), window=rng.randint(0, 2))
        if kind == "attention":
            c["norm"] = rng.choice(["none", "layer", "rms"])
            c["lse"] = rng.random() < 0.2
        if kind in ("host", "plan"):
            c["B"], c["layout"] = 1, "HND"
        nb = _blocks(c)
        elems = c["B"] * c["H"] * _tokens(c) * D
        if elems > _MAX_ELEMS or c["B"] * c["H"] * nb * nb * _kept_share(c) * D > _MAX_WALK:
            continue
        if c["H"] * nb * nb > _MAX_MASK or (kind == "host" and elems > _MAX_ELEMS // 4):
            continue
        return c


def _tokens(c):
    return c["n_text"] + c["F"] * c["Y"] * c["X"]


def _blocks(c):
    return (_tokens(c) + BLOCK - 1) // BLOCK


def _text_blocks(c):
    return (c["n_text"] + BLOCK - 1) // BLOCK


def _kept_share(c):
    """Expected share of kept blocks: text rows and columns and the band in full, the rest at the density."""
    nb, t, w = _blocks(c), _text_blocks(c), c["window"]
    text = nb * nb - (nb - t) * (nb - t)
    v = nb - t
    band = sum(min(v - 1, i + w) - max(0, i - w) + 1 for i in range(v))
    return (text + band + c["density"] * (v * v - band)) / (nb * nb)


def _list_capacity(c):
    """Entries that hold the list of any drawn mask of the case: the expected number of kept blocks and nine deviations."""
    n = c["H"] * _blocks(c) ** 2
    return int(n * _kept_share(c) + 4.5 * math.sqrt(n)) + 64


def _mask(c, gen):
    nb, t = _blocks(c), _text_blocks(c)
    m = torch.rand(c["H"], nb, nb, generator=gen, device="cuda") < c["density"]
    i = torch.arange(nb, device="cuda")
    m |= ((i.view(-1, 1) - i.view(1, -1)).abs() <= c["window"]).unsqueeze(0)
    if t:
        m[:, :t, :] = True
        m[:, :, :t] = True
    return m


def _activations(c, gen):
    B, H, N, D, dt = c["B"], c["H"], _tokens(c), c["D"], DTYPES[c["dtype"]]
    nhd = c["layout"] == "NHD"
    shape = (B, N, H, D) if nhd else (B, H, N, D)
    q = torch.randn(shape, generator=gen, device="cuda").to(dt)
    k = torch.randn(shape, generator=gen, device="cuda")
    k += math.sqrt(2.0) * torch.randn((1, 1, H, D) if nhd else (1, H, 1, D), generator=gen, device="cuda")
    v = torch.randn(shape, generator=gen, device="cuda").to(dt)
    return q, k.to(dt), v


def _norm(c, gen):
    if c["norm"] == "none":
        return None
    n = c["D"] if c["norm"] == "layer" else c["H"] * c["D"]
    dt = DTYPES[c["dtype"]]
    weight = (1 + 0.1 * torch.randn(n, generator=gen, device="cuda")).to(dt)
    bias = (0.1 * torch.randn(n, generator=gen, device="cuda")).to(dt) if c["norm"] == "layer" else None
    return pb.QKNorm(c["norm"], weight, bias, 1e-6)


def prepare(case, seed):
    c = case
    gen = torch.Generator(device="cuda").manual_seed(seed)
    grid = (c["F"], c["Y"], c["X"])
    s = {"case": c, "grid": grid}
    if c["kind"] == "plan":
        s["mask"] = _mask(c, gen)
        return s
    if c["kind"] == "merge":
        a, b, _ = _activations(c, gen)
        lse = 6 + torch.randn(2, c["B"], c["H"], _tokens(c), generator=gen, device="cuda")
        lse[torch.rand(lse.shape, generator=gen, device="cuda") < 0.01] = -math.inf     # rows without a kept block in one part
        s.update(a=a, b=b, lse_a=lse[0].contiguous(), lse_b=lse[1].contiguous())
        return s
    s["q"], s["k"], s["v"] = _activations(c, gen)
    if c["kind"] == "operator":
        s["mask"] = _mask(c, gen)
        return s
    orders = torch.randint(0, 6, (c["H"],), generator=gen, device="cuda", dtype=torch.int32)
    s["rope"] = pb.rope_tables(grid, c["D"], c["family"]) if c["family"] != "none" else None
    if c["kind"] == "host":
        shape = tuple(s["q"].shape)
        for name in ("q", "k", "v"):
            host = pb.pinned_like(shape, s[name].dtype)
            host.copy_(s[name])
            s[name] = host
        s["out"] = pb.pinned_like(shape, s["q"].dtype)
        s["handle"] = pb.HostPipelinedAttention(orders.cpu(), _mask(c, gen), shape, s["q"].dtype, grid_fhw=grid,
                                                n_text=c["n_text"], rope=s["rope"])
        return s
    s["pplan"] = pb.PermutePlan({"permute": orders.view(1, -1)}, grid)
    if c["kind"] == "attention":
        s["plan"] = pb.compact_plan(_mask(c, gen), pairing="overlap")
        s["q_norm"], s["k_norm"] = _norm(c, gen), _norm(c, gen)
    return s


def run(state):
    s = state
    c = s["case"]
    kind = c["kind"]
    if kind == "attention":
        return pb.paro_attention(s["q"], s["k"], s["v"], s["pplan"], s["plan"], i_block=0, grid_fhw=s["grid"],
                                 n_text=c["n_text"], rope=s["rope"], tensor_layout=c["layout"], return_lse=c["lse"],
                                 q_norm=s["q_norm"], k_norm=s["k_norm"])
    if kind == "operator":
        return pb.paroattn_qk_int8_pv_fp16_cuda(s["q"], s["k"], s["v"], s["mask"], tensor_layout=c["layout"])
    if kind == "prep":
        orders, lay = s["pplan"].orders(0), c["layout"]
        q8, qs, _ = pb.prep_qk_int8(s["q"], orders, s["grid"], c["n_text"], s["rope"], group=32, tensor_layout=lay)
        k8, ks, km = pb.prep_qk_int8(s["k"], orders, s["grid"], c["n_text"], s["rope"], group=64, smooth=True,
                                     tensor_layout=lay)
        v16, vs, vm, _ = pb.prep_v_fp8(s["v"], orders, s["grid"], c["n_text"], tensor_layout=lay)
        return q8, qs, k8, ks, km, v16, vs, vm
    if kind == "plan":
        p = pb.compact_plan(s["mask"], pairing="overlap")
        # the lists are as long as the mask has kept blocks: they are returned at the length of a buffer that holds any mask's
        cap, prows = _list_capacity(c), c["H"] * ((p.nbq + 1) // 2)
        out = {name: torch.nn.functional.pad(t, (0, cap - t.numel()))
               for name, t in (("cols", p.cols), ("pair_ent", p.pair_ent), ("sched", p.sched))}
        pair_q = p.pair_q if p.pair_q is not None else torch.full((prows, 2), -1, dtype=torch.int32, device="cuda")
        kernel = p.sched_cnt_kernel if p.sched_cnt_kernel is not None else p.sched_cnt
        return dict(out, row_ptr=p.row_ptr, pair_ptr=p.pair_ptr, sched_cnt=p.sched_cnt, pair_q=pair_q,
                    sched_cnt_kernel=kernel)
    if kind == "merge":
        return pb.merge_attention_states(s["a"], s["lse_a"], s["b"], s["lse_b"], tensor_layout=c["layout"])
    return s["handle"](s["q"], s["k"], s["v"], s["out"])


def work(case):
    c = case
    nb, N = _blocks(c), _tokens(c)
    rows = c["B"] * c["H"] * N
    elems = rows * c["D"]
    kept = round(c["H"] * nb * nb * _kept_share(c))             # blocks of the mask; every batch entry walks them
    if c["kind"] == "plan":
        # the mask once; what the kernel walks (a 2-byte k-block id per kept block and half); all overlaps of two rows
        return {"bytes": c["H"] * nb * nb + 2 * kept, "flops": c["H"] * nb * nb * nb}
    if c["kind"] == "merge":
        return {"bytes": 6 * elems + 12 * rows, "flops": 3 * elems}
    if c["kind"] == "prep":
        return {"bytes": 6 * elems + 4 * elems, "flops": 10 * elems}   # three 16-bit tensors in; int8 Q, K, bf16 V out
    mask = c["H"] * nb * nb if c["kind"] == "operator" else 2 * kept
    return {"bytes": 8 * elems + mask + (4 * rows if c["lse"] else 0), "flops": c["B"] * kept * 4 * BLOCK * BLOCK * c["D"]}


def tolerance(case):
    if case["kind"] in ("plan", "prep"):
        return "exact"       # lists, INT8 and e4m3 values, their scales and the channel means are specified bit for bit
    bf16 = case["dtype"] == "bf16"
    if case["kind"] == "merge":
        return {"rel": 6e-3 if bf16 else 8e-4}     # the result's rounding; against fp64: 1.6e-3, 2.0e-4
    # 16-bit P and output; the online-softmax walk against the fixed-reference walk: up to 4.9e-4, 2.0e-4
    return {"rel": 2e-3 if bf16 else 1e-3}
