"""Workloads of this package as a user's program runs them: single structured linears through the public operator
functions, and the three networks built on them.  Each case is a dict of plain values:

  kind      operator or network (see CALLS and NETWORKS)
  inp, out  features of the linear; b blocks per side, rank
  tokens    rows of x
  dtype     "fp16" | "bf16"
  bits, group   weight-quantised BLAST: int8 | packed int4 factors, a scale per output channel (0) or per 128 indices
  batch     sequences / images / latents of a network step;  layers its depth;  method its linears

Sizes: the Llama-7B, ViT-B/16 and DiT-XL/2 linears with the ranks that halve their parameters, and generic ones.
"""
import math

import torch

import mem_efficient_blr_b200.blast_kernels as bk
import mem_efficient_blr_b200.blast_sym_quant_kernels as bq
import mem_efficient_blr_b200.low_rank_kernels as lk
import mem_efficient_blr_b200.monarch_kernels as mk
from mem_efficient_blr_b200 import networks as nw

DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16}
NETWORKS = ("llama_decode", "vit", "dit")
CACHE = 2048  # key/value slots of the decoder, all in use


def _linear(kind, inp, out, b, rank, tokens, dtype, **more):
    return dict(kind=kind, inp=inp, out=out, b=b, rank=rank, tokens=tokens, dtype=dtype, **more)


def listed():
    cases = {
        # one new token of one sequence: the headline layer (gate_proj) with int8 factors, per-channel scales
        "wq int8 gate 1 tok": _linear("wq", 4096, 11008, 16, 1024, 1, "fp16", bits=8, group=0),
        # the same layer with packed int4 factors, a batch of 16 sequences (the largest decode-size call)
        "wq int4 gate 16 tok": _linear("wq", 4096, 11008, 16, 1024, 16, "fp16", bits=4, group=0),
        # int8 factors kept as the only copy of the layer, a short ragged prompt
        "wq int8 gate 333 tok": _linear("wq", 4096, 11008, 16, 1024, 333, "fp16", bits=8, group=0),
        # attention projection in the torch layouts, 4 sequences decoding
        "blast q_proj 4 tok": _linear("torch", 4096, 4096, 16, 1024, 4, "fp16"),
        # drop-in call of the reference's Llama configuration (Triton-entry layouts, bf16), decode, long input
        "blast partial down 1 tok": _linear("partial", 11008, 4096, 16, 1488, 1, "bf16"),
        # the single-layer benchmark of the project: 128 tokens through gate_proj
        "blast gate 128 tok": _linear("torch", 4096, 11008, 16, 1024, 128, "fp16"),
        # prefill of a 2048-token prompt, drop-in layouts and dtype
        "blast partial gate 2048 tok": _linear("partial", 4096, 11008, 16, 1488, 2048, "bf16"),
        # the other two structured families of the layer sweep, drop-in layouts
        "monarch gate 128 tok": _linear("monarch", 4096, 11008, 4, 1536, 128, "bf16"),
        "low rank down 16 tok": _linear("low_rank", 11008, 4096, 1, 1024, 16, "bf16"),
        # decoder layers, one token step of 4 sequences at a full cache, replayed from a CUDA graph as a server does
        "llama decode batch 4": dict(kind="llama_decode", batch=4, layers=4, method="blast"),
        # image encoder, called eagerly on a batch of images
        "vit batch 16": dict(kind="vit", batch=16, layers=12, method="blast"),
        # denoiser, one of many steps of equal shape, replayed from a CUDA graph
        "dit step batch 8": dict(kind="dit", batch=8, layers=28, method="blast"),
    }
    return [dict(c, name=n) for n, c in cases.items()]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("torch", "torch", "partial", "partial", "bmm", "wq", "wq", "wq", "monarch", "monarch", "low_rank", "low_rank")
                      + NETWORKS)
    if kind in NETWORKS:
        most, layers = {"llama_decode": (16, 4), "vit": (32, 12), "dit": (8, 28)}[kind]
        method = rng.choice(("blast", "blast_int8")) if kind == "llama_decode" else "blast"
        return dict(kind=kind, batch=_log_int(rng, 1, most), layers=layers, method=method)
    tokens = _log_int(rng, 1, 4096)
    dtype = rng.choice(("fp16", "bf16"))
    if rng.random() < 0.6:  # the linears of the networks
        inp, out, b, rank = rng.choice(((4096, 4096, 16, 1024), (4096, 11008, 16, 1024), (4096, 11008, 16, 1488), (11008, 4096, 16, 1488),
                                        (768, 2304, 16, 256), (768, 3072, 16, 288), (3072, 768, 16, 288), (1152, 3456, 9, 384),
                                        (1152, 4608, 9, 256)))
    else:                   # generic ones, odd multiples of the block widths among them
        b, step = rng.choice((4, 6, 8, 16)), 32 if kind == "wq" else 8
        inp, out = (b * step * _log_int(rng, 128 // step, 6144 // (b * step)) for _ in range(2))
        rank = step * _log_int(rng, 128 // step, 1536 // step)
    more = {}
    if kind == "wq":
        wide = (inp // b) % 32 == 0 and rank % 32 == 0
        more["bits"] = rng.choice((8, 4)) if wide else 8
        more["group"] = 128 if (inp // b) % 128 == 0 and rank % 128 == 0 and rng.random() < 0.3 else 0
    elif kind == "monarch":
        b = rng.choice((4, 16)) if (inp % 128, out % 128) == (0, 0) else 4
        inp, out = inp // (8 * b) * 8 * b, out // (8 * b) * 8 * b
        rank = max(8 * b, rank // (8 * b) * 8 * b)
    elif kind == "low_rank":
        b = 1
    return _linear(kind, inp, out, b, rank, tokens, dtype, **more)


# ------------------------------------------------------------------------------------------------------------- inputs
def _linear_state(c, gen):
    dt = DTYPES[c["dtype"]]
    b, R, P, Q = c["b"], c["rank"], c["inp"] // c["b"], c["out"] // c["b"]

    def normal(*shape, fan=1.0):
        return (torch.randn(*shape, generator=gen, device="cuda") / math.sqrt(fan)).to(dt)

    x = normal(c["tokens"], c["inp"])
    kind = c["kind"]
    if kind == "monarch":    # w1 (b, P, rank), w2 (b, Q, rank)
        return (mk.triton_monarch_right_fp16, (x, normal(b, P, R, fan=P), normal(b, Q, R, fan=R)))
    if kind == "low_rank":   # (I, R), (R, O)
        return (lk.triton_low_rank_fp16, (x, normal(c["inp"], R, fan=c["inp"]), normal(R, c["out"], fan=R)))
    # variance-preserving BLAST factors: S ~ U(0.5, 1.5)
    S = torch.rand(b, b, R, generator=gen, device="cuda").add_(0.5).to(dt)
    fan_u = R * b * 13.0 / 12.0
    if kind == "partial":    # U (b, R, Q), V (b, P, R), S (b_in, b_out, R)
        return (bk.triton_blast_partial_grouped_fp16, (x, normal(b, R, Q, fan=fan_u), normal(b, P, R, fan=P), S))
    if kind == "bmm":        # U (b, Q, R), V (b, P, R), S (R, b_out, b_in)
        return (bk.triton_blast_bmm_fp16, (x, normal(b, Q, R, fan=fan_u), normal(b, P, R, fan=P), S.permute(2, 0, 1).contiguous()))
    U, Vt = normal(b, Q, R, fan=fan_u), normal(b, R, P, fan=P)
    if kind == "torch":
        return (bk.blast_torch_layout, (x, U, Vt, S))
    Uq, us, Vq, vs = bq.quantize_blast_factors(U, Vt, c["bits"], c["group"])
    return (bq.blast_wq, (x, Uq, us, Vq, vs, S, c["bits"], c["group"]))


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    if case["kind"] not in NETWORKS:
        fn, args = _linear_state(case, gen)
        return {"kind": "linear", "fn": fn, "args": args}
    torch.manual_seed(seed)  # (torch's own layers inside the networks draw from the global generators)
    B, kind = case["batch"], case["kind"]
    half = torch.float16
    if kind == "llama_decode":
        shape = nw.LlamaShape(layers=case["layers"])
        model = nw.LlamaDecoder(shape, case["method"], batch=B, cache_len=CACHE, dtype=half, seed=seed, init_on_device=True)
        for t in model.kcache + model.vcache:
            t.normal_(0, 0.5, generator=gen)
        ids = torch.randint(0, shape.vocab, (B, 1), generator=gen, device="cuda")
        pos = torch.tensor([CACHE - 1], device="cuda")
        step = nw.GraphedCall(model.decode_step, ids.clone(), pos.clone())
        return {"kind": kind, "model": model, "call": step, "inputs": (ids, pos)}
    if kind == "vit":
        shape = nw.ViTShape(layers=case["layers"])
        model = nw.ViTEncoder(shape, case["method"], dtype=half, seed=seed, init_on_device=True)
        img = torch.randn(B, 3, shape.image, shape.image, generator=gen, device="cuda").to(half)
        return {"kind": kind, "model": model, "call": model, "inputs": (img,)}
    shape = nw.DiTShape(layers=case["layers"])
    model = nw.DiTDenoiser(shape, case["method"], dtype=half, seed=seed, init_on_device=True)
    lat = torch.randn(B, shape.channels, shape.latent, shape.latent, generator=gen, device="cuda").to(half)
    t = torch.randint(0, 1000, (B,), generator=gen, device="cuda")
    y = torch.randint(0, shape.classes, (B,), generator=gen, device="cuda")
    step = nw.GraphedCall(model, lat.clone(), t.clone(), y.clone())
    return {"kind": kind, "model": model, "call": step, "inputs": (lat, t, y)}


def run(state):
    if state["kind"] == "linear":
        return state["fn"](*state["args"])
    out = state["call"](*state["inputs"])
    if state["kind"] == "llama_decode":  # the step writes the new token's keys and values into the caches
        return {"logits": out, "k": state["model"].kcache, "v": state["model"].vcache}
    return out


# --------------------------------------------------------------------------------------------------------------- work
def _layer_work(n, inp, out, b, R, bits=16, group=0, coupled=True):
    """(bytes of the weights, flops) of one structured linear on n rows."""
    nbytes = bits / 8 * R * (inp + out)
    if bits != 16:  # fp16 scales: one per weight row, or one per group of a row
        nbytes += 2.0 * R * (inp + out) / group if group else 2.0 * (b * R + out)
    flops = 2.0 * n * R * (inp + out)
    if coupled:
        nbytes += 2.0 * b * b * R
        flops += 2.0 * n * b * b * R
    return nbytes, flops


def _dense_work(n, inp, out):
    return 2.0 * inp * out, 2.0 * n * inp * out


def work(case):
    kind = case["kind"]
    if kind not in NETWORKS:
        n = case["tokens"]
        nb, fl = _layer_work(n, case["inp"], case["out"], case["b"], case["rank"], case.get("bits", 16), case.get("group", 0),
                             coupled=kind not in ("monarch", "low_rank"))
        return {"bytes": nb + 2.0 * n * (case["inp"] + case["out"]), "flops": fl}
    B, L = case["batch"], case["layers"]
    bits = 8 if case["method"] == "blast_int8" else 16
    if kind == "llama_decode":
        s = nw.LlamaShape(layers=L)
        per = [_layer_work(B, s.d, s.d, s.b, s.rank_attn, bits)] * 4 + [_layer_work(B, s.d, s.ffn, s.b, s.rank_mlp, bits)] * 2 \
            + [_layer_work(B, s.ffn, s.d, s.b, s.rank_mlp, bits), (2.0 * 2 * B * CACHE * s.d, 4.0 * B * CACHE * s.d)]
        once = [_dense_work(B, s.d, s.vocab), (2.0 * B * (s.d + s.vocab), 0.0)]
    elif kind == "vit":
        s, T = nw.ViTShape(layers=L), B * 197
        per = [_layer_work(T, s.d, 3 * s.d, s.b, s.ranks["qkv"], bits), _dense_work(T, s.d, s.d),
               _layer_work(T, s.d, s.mlp, s.b, s.ranks["intermediate"], bits), _layer_work(T, s.mlp, s.d, s.b, s.ranks["output"], bits),
               (0.0, 4.0 * T * 197 * s.d)]
        once = [_dense_work(B * 196, 3 * s.patch ** 2, s.d), (2.0 * (B * 3 * s.image ** 2 + T * s.d), 0.0)]
    else:
        s, T = nw.DiTShape(layers=L), B * 256
        per = [_layer_work(T, s.d, 3 * s.d, s.b, s.ranks["qkv"], bits), _dense_work(T, s.d, s.d),
               _layer_work(T, s.d, s.mlp, s.b, s.ranks["fc1"], bits), _dense_work(T, s.mlp, s.d),
               _layer_work(B, s.d, 6 * s.d, s.b, s.ranks["adaln"], bits), (0.0, 4.0 * T * 256 * s.d)]
        once = [_dense_work(B, s.d, 2 * s.d), _dense_work(B, s.d, s.d), (2.0 * B * s.latent ** 2 * 3 * s.channels, 0.0)]
    return {"bytes": L * sum(p[0] for p in per) + sum(p[0] for p in once), "flops": L * sum(p[1] for p in per) + sum(p[1] for p in once)}


def tolerance(case):
    """fp32 accumulation on 16-bit factors, the intermediates and the result rounded to 16 bits (11 | 8 bits of mantissa);
    a network chains a few dozen such layers."""
    if case["kind"] in NETWORKS:
        return {"rel": 1e-2}
    return {"rel": 2e-3 if case["dtype"] == "fp16" else 1e-2}
