"""What a user of this framework has it do, as cases that can be timed and compared.

Four kinds of calls, through the package's public entry points:

  host      one product with host arrays (Backend.gemm): the drop-in call behind zen::quant::gemv / gemm, PCIe included
  layer     a decoder layer's projections on resident tensors, q|k|v, o, gate|up, down (Backend.dev_gemv): what a caller that
            keeps its activations on the device does for every token, or for a block of up to eight to verify
  head      the output projection over the vocabulary and the greedy pick behind it
  block     one product of a block of tokens on the tensor cores (Backend.dev_gemm_*): a prompt through one matrix
  request   a whole request through a decoder (LlamaDecoder, KipiraxDecoder, SikivikDecoder): reset, prompt, greedy tokens

Sizes are those of the repository's benchmark (a Llama-3-8B layer, its vocabulary and prompt; decoders of width 1024 to 4096) and
others of the same ranges.  Decoders have two to four layers: every layer is alike.  Weights are made up.  A made-up model's head
answers each token's embedding with one certain successor, as a trained model is sure of most tokens: with a random head the greedy
pick would be decided by rounding.
"""
import math

import numpy as np
import torch

from zeninfer_b200 import Backend
from zeninfer_b200.backend import ACT_FP32, ACT_INT8
from zeninfer_b200.kipirax import KipiraxConfig, KipiraxDecoder
from zeninfer_b200.kipirax import random_tensor as kipirax_tensor
from zeninfer_b200.kipirax import tensor_plan as kipirax_plan
from zeninfer_b200.llama import LlamaConfig, LlamaDecoder
from zeninfer_b200.llama import tensor_plan as llama_plan
from zeninfer_b200.sikivik import SikivikConfig, SikivikDecoder
from zeninfer_b200.sikivik import random_tensor as sikivik_tensor
from zeninfer_b200.sikivik import tensor_plan as sikivik_plan

FORMATS = ("Q8_0", "Q4_0", "Q6_K", "Q4_K", "Q5_K")
BLOCK = {"Q8_0": (32, 34), "Q4_0": (32, 18), "Q6_K": (256, 210), "Q4_K": (256, 144), "Q5_K": (256, 176)}     # weights, bytes of a block
MODES = {"int8": ACT_INT8, "fp32": ACT_FP32}
HIDDEN = {1024: 4096, 2048: 8192, 4096: 14336}       # width of a decoder -> its feed-forward
F64 = torch.float64
DEV = "cuda"


# ---- the cases ---------------------------------------------------------------------------------------------------------

def listed():
    return [
        # a plug-in's single product: the smallest call, latency counts
        dict(name="host q8_0 4096x4096", kind="host", fmt="Q8_0", act="int8", tokens=1, rows=4096, columns=4096),
        # a token through an 8B layer's projections, in the default format and in the small ones
        dict(name="layer q8_0 1 token", kind="layer", fmt="Q8_0", act="int8", tokens=1, width=4096, kv=1024, ff=14336),
        dict(name="layer q4_0 1 token", kind="layer", fmt="Q4_0", act="fp32", tokens=1, width=4096, kv=1024, ff=14336),
        dict(name="layer q4_k 1 token", kind="layer", fmt="Q4_K", act="fp32", tokens=1, width=4096, kv=1024, ff=14336),
        # the head of a speculative-verify block
        dict(name="head q6_k 8 tokens", kind="head", fmt="Q6_K", act="fp32", tokens=8, vocab=128256, width=4096),
        # a prompt block through the up projection, and a short ragged one in a small format
        dict(name="block q8_0 512 tokens", kind="block", fmt="Q8_0", act="int8", tokens=512, rows=14336, columns=4096),
        dict(name="block q4_k 77 tokens", kind="block", fmt="Q4_K", act="fp32", tokens=77, rows=11008, columns=4096),
        # requests: a small model answering a short question, an 8B layer pair with a prompt and an answer, a long document
        dict(name="llama 1024 short", kind="request", arch="llama", act="fp32", width=1024, layers=4, vocab=32000, prompt=9, new=48),
        dict(name="llama 4096", kind="request", arch="llama", act="int8", width=4096, layers=2, vocab=32000, prompt=512, new=32),
        dict(name="llama 4096 long", kind="request", arch="llama", act="int8", width=4096, layers=2, vocab=32000, prompt=2000, new=4),
        # the bf16 decoders
        dict(name="kipirax 2048", kind="request", arch="kipirax", act="bf16", width=2048, layers=4, vocab=32000, prompt=512, new=32),
        dict(name="sikivik 4096", kind="request", arch="sikivik", act="bf16", width=4096, layers=4, vocab=32000, prompt=301, new=32),
    ]


def _spread(rng, low, high, multiple=1):
    """A size from low to high, even over its logarithm."""
    n = int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))
    return min(max(n // multiple * multiple, low), high)


def draw(rng):
    kind = rng.choice(("host", "layer", "head", "block", "request", "request", "request"))
    fmt = rng.choice(FORMATS)
    act = rng.choice(("int8", "fp32")) if fmt == "Q8_0" else "fp32"
    if kind == "host":
        return dict(kind=kind, fmt=fmt, act=act, tokens=rng.choice((1, 1, 2, 5, 8, 13)), rows=_spread(rng, 256, 8192), columns=_spread(rng, 1024, 8192, 256))
    if kind == "layer":
        width = rng.choice((1024, 2048, 3072, 4096))
        return dict(kind=kind, fmt=fmt, act=act, tokens=rng.choice((1, 1, 1, 2, 4, 8)), width=width, kv=width // rng.choice((1, 2, 4)),
                    ff=_spread(rng, 2 * width, 14336, 256))
    if kind == "head":
        fmt = rng.choice(("Q6_K", "Q8_0"))
        return dict(kind=kind, fmt=fmt, act="fp32", tokens=rng.choice((1, 1, 3, 8)), vocab=rng.choice((32000, 50257, 128256)), width=rng.choice((2048, 4096)))
    if kind == "block":
        return dict(kind=kind, fmt=fmt, act=act, tokens=_spread(rng, 16, 1024), rows=_spread(rng, 1024, 14336), columns=_spread(rng, 1024, 14336, 256))
    arch, width = rng.choice(("llama", "kipirax", "sikivik")), rng.choice((1024, 2048, 4096))
    return dict(kind=kind, arch=arch, act=rng.choice(("int8", "fp32")) if arch == "llama" else "bf16", width=width, layers=2 if width == 4096 else 4,
                vocab=rng.choice((16384, 32000)), prompt=_spread(rng, 5, 1400), new=_spread(rng, 4, 32))


# ---- made-up weights as file blocks, on the device --------------------------------------------------------------------------

def _generator(seed, part):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed * 1000003 + part)
    return g


def _half_bytes(t):
    return t.to(torch.float16).contiguous().view(torch.uint8).view(*t.shape, 2)


def _pack(fmt, w):
    """fp32 [rows, K] on the device -> the format's raw rows, uint8 [rows, bytes].  Q4_K / Q5_K: one scale and minimum per 32 weights."""
    rows, k = w.shape
    per, size = BLOCK[fmt]
    n = rows * k // per
    out = torch.empty((n, size), dtype=torch.uint8, device=w.device)
    b = w.view(n, per)
    if fmt == "Q8_0":
        d = b.abs().amax(1) / 127.0
        out[:, 0:2] = _half_bytes(d)
        out[:, 2:] = torch.round(b / d.clamp_min(1e-30)[:, None]).clamp_(-127, 127).to(torch.int8).view(torch.uint8)
    elif fmt == "Q4_0":
        d = b.abs().amax(1) / 8.0
        q = torch.round(b / d.clamp_min(1e-30)[:, None] + 8.0).clamp_(0, 15).to(torch.uint8)
        out[:, 0:2] = _half_bytes(d)
        out[:, 2:] = q[:, :16] | (q[:, 16:] << 4)
    elif fmt == "Q6_K":
        group = b.view(n, 16, 16)
        scale = group.abs().amax(2) / 31.0
        d = (scale.amax(1) / 127.0).to(torch.float16)
        sc = torch.round(scale / d.float().clamp_min(1e-30)[:, None]).clamp_(1, 127)
        q = (torch.round(group / (d.float()[:, None] * sc).clamp_min(1e-30)[..., None]).clamp_(-32, 31) + 32).to(torch.uint8).view(n, 2, 4, 32)
        ql, qh = out[:, :128].view(n, 2, 2, 32), out[:, 128:192].view(n, 2, 32)
        ql[:, :, 0] = (q[:, :, 0] & 15) | ((q[:, :, 2] & 15) << 4)
        ql[:, :, 1] = (q[:, :, 1] & 15) | ((q[:, :, 3] & 15) << 4)
        qh[:] = (q[:, :, 0] >> 4) | ((q[:, :, 1] >> 4) << 2) | ((q[:, :, 2] >> 4) << 4) | ((q[:, :, 3] >> 4) << 6)
        out[:, 192:208] = sc.to(torch.int8).view(torch.uint8)
        out[:, 208:210] = _half_bytes(d)
    else:
        top = 31.0 if fmt == "Q5_K" else 15.0
        sub = b.view(n, 8, 32)
        low, high = sub.amin(2).clamp_max(0.0), sub.amax(2)
        scale, minimum = (high - low).clamp_min(0.0) / top, -low
        d, dmin = (scale.amax(1) / 63.0).to(torch.float16), (minimum.amax(1) / 63.0).to(torch.float16)
        sc = torch.round(scale / d.float().clamp_min(1e-30)[:, None]).clamp_(0, 63)
        mn = torch.round(minimum / dmin.float().clamp_min(1e-30)[:, None]).clamp_(0, 63)
        q = torch.round((sub + (dmin.float()[:, None] * mn)[..., None]) / (d.float()[:, None] * sc).clamp_min(1e-30)[..., None]).clamp_(0, top).to(torch.uint8)
        s, m = sc.to(torch.uint8), mn.to(torch.uint8)
        out[:, 0:2], out[:, 2:4] = _half_bytes(d), _half_bytes(dmin)
        out[:, 4:8] = s[:, :4] | ((s[:, 4:] >> 4) << 6)
        out[:, 8:12] = m[:, :4] | ((m[:, 4:] >> 4) << 6)
        out[:, 12:16] = (s[:, 4:] & 15) | ((m[:, 4:] & 15) << 4)
        pairs = q.view(n, 4, 2, 32)
        out[:, size - 128:] = ((pairs[:, :, 0] & 15) | ((pairs[:, :, 1] & 15) << 4)).view(n, 128)
        if fmt == "Q5_K":
            out[:, 16:48] = sum((q[:, j] >> 4) << j for j in range(8))
    return out.view(rows, -1)


def _unpack(fmt, raw, k):
    """What the blocks say, in 64 bits."""
    rows = raw.shape[0]
    per, size = BLOCK[fmt]
    b = raw.view(-1, size)
    n = b.shape[0]
    half = lambda a, c: b[:, a:c].contiguous().view(torch.float16).to(F64)
    if fmt == "Q8_0":
        w = b[:, 2:].contiguous().view(torch.int8).to(F64) * half(0, 2)
    elif fmt == "Q4_0":
        w = (torch.cat([b[:, 2:] & 15, b[:, 2:] >> 4], 1).to(F64) - 8.0) * half(0, 2)
    elif fmt == "Q6_K":
        ql, qh = b[:, :128].reshape(n, 2, 2, 32), b[:, 128:192].reshape(n, 2, 32)
        low = torch.cat([ql & 15, ql >> 4], 2)
        high = torch.stack([(qh >> (2 * i)) & 3 for i in range(4)], 2)
        q = (low | (high << 4)).to(F64).view(n, 16, 16) - 32.0
        w = q * (half(208, 210) * b[:, 192:208].contiguous().view(torch.int8).to(F64))[..., None]
    else:
        s = b[:, 4:16]
        sc = torch.cat([s[:, :4] & 63, (s[:, 8:] & 15) | ((s[:, :4] >> 6) << 4)], 1).to(F64)
        mn = torch.cat([s[:, 4:8] & 63, (s[:, 8:] >> 4) | ((s[:, 4:8] >> 6) << 4)], 1).to(F64)
        nib = b[:, size - 128:].reshape(n, 4, 32)
        q = torch.stack([nib & 15, nib >> 4], 2).view(n, 8, 32)
        if fmt == "Q5_K":
            q = q | (torch.stack([(b[:, 16:48] >> j) & 1 for j in range(8)], 1) << 4)
        w = q.to(F64) * (half(0, 2) * sc)[..., None] - (half(2, 4) * mn)[..., None]
    return w.view(rows, k)


def _matrix(fmt, rows, columns, seed, part):
    return _pack(fmt, torch.randn((rows, columns), generator=_generator(seed, part), device=DEV) * columns ** -0.5)


def _acts(tokens, columns, seed):
    return torch.randn((tokens, columns), generator=_generator(seed, 999), device=DEV)


def _int8_codes(x):
    """Activations as the int8 route takes them, a scale per 32 values: the values the codes stand for, in 64 bits."""
    b = x.float().reshape(-1, 32)
    d = b.abs().amax(1, keepdim=True) / 127.0
    v = (b * torch.where(d > 0, 1.0 / d, torch.zeros_like(d))).clamp(-127.0, 127.0)
    t = torch.trunc(v)
    q = t + torch.where((v - t).abs() >= 0.5, torch.sign(v), torch.zeros_like(v))
    return (q.to(F64) * d.to(F64)).view(x.shape)


# ---- products -------------------------------------------------------------------------------------------------------------

_the_backend = None


def _backend():
    global _the_backend
    if _the_backend is None:
        _the_backend = Backend()
    return _the_backend


class Held:
    """What a program keeps: resident tensors, a decoder, host arrays the backend knows by address."""

    def __init__(self, case):
        self.case, self.handles, self.decoder, self.known = case, [], None, []

    def upload(self, fmt, raw, columns):
        h = _backend().dev_upload(fmt, raw.cpu().numpy(), raw.shape[0], columns)
        self.handles.append(h)
        return h

    def __del__(self):
        if self.decoder is not None:
            self.decoder.close()
        for h in self.handles:
            _backend().dev_free(h)
        for a in self.known:
            _backend().release_weights(a)


def _layer_products(case):
    """(rows of the tensors that share an input, their columns) of every launch."""
    w, kv, ff = case["width"], case["kv"], case["ff"]
    return [([w, kv, kv], w), ([w], w), ([ff, ff], w), ([w], ff)]


def _case_products(case):
    return {"host": lambda: [([case["rows"]], case["columns"])], "block": lambda: [([case["rows"]], case["columns"])],
            "layer": lambda: _layer_products(case), "head": lambda: [([case["vocab"]], case["width"])]}[case["kind"]]()


def _prepare_products(case, seed):
    be, s, fmt, tokens = _backend(), Held(case), case["fmt"], case["tokens"]
    s.launches = []
    part = 0
    for rows, columns in _case_products(case):
        x = _acts(tokens, columns, seed + part)
        handles = []
        for r in rows:
            raw = _matrix(fmt, r, columns, seed, part)
            part += 1
            if case["kind"] == "host":
                s.known.append(raw.cpu().numpy())
            else:
                handles.append(s.upload(fmt, raw, columns))
        s.launches.append((handles, x, [torch.empty((tokens, r), device=DEV) for r in rows], columns, rows))
    if case["kind"] == "host":
        be.set_q8_act_mode(MODES[case["act"]])
        s.x = s.launches[0][1].cpu().numpy()
    if case["kind"] == "head":
        s.pick = torch.empty(tokens, dtype=torch.int64, device=DEV)
    if case["kind"] == "block" or (case["kind"] == "head" and fmt == "Q6_K" and tokens >= 7):
        rows, columns = s.launches[0][4][0], s.launches[0][3]
        need = {"Q8_0": lambda: be.gemm_workspace_bytes(tokens, columns, MODES[case["act"]]), "Q6_K": lambda: be.gemm_q6_k_workspace_bytes(tokens, columns),
                "Q4_0": lambda: be.gemm_q4_0_workspace_bytes(tokens, rows, columns)}.get(fmt, lambda: be.gemm_kquant_workspace_bytes(tokens, rows, columns))()
        s.workspace = torch.empty(need, dtype=torch.uint8, device=DEV)
    else:
        s.workspace = None
    return s


def _run_products(s):
    be, case = _backend(), s.case
    fmt, tokens, stream = case["fmt"], case["tokens"], torch.cuda.current_stream().cuda_stream
    if case["kind"] == "host":
        return be.gemm(fmt, s.known[0], s.x, tokens, case["rows"], case["columns"])
    if s.workspace is not None:
        (h,), x, (y,), _, _ = s.launches[0]
        rest = (y.data_ptr(), x.data_ptr(), tokens, s.workspace.data_ptr(), s.workspace.numel(), stream)
        if fmt == "Q8_0":
            be.dev_gemm_q8_0([h], [y.data_ptr()], *rest[1:], act_mode=MODES[case["act"]])
        else:
            {"Q6_K": be.dev_gemm_q6_k, "Q4_0": be.dev_gemm_q4_0}.get(fmt, be.dev_gemm_kquant)(h, *rest)
    else:
        for handles, x, ys, _, _ in s.launches:
            be.dev_gemv(handles, [y.data_ptr() for y in ys], x.data_ptr(), tokens, MODES[case["act"]], stream)
    if case["kind"] == "head":
        logits = s.launches[0][2][0]
        be.dev_greedy_pick([(logits.data_ptr(), case["vocab"], 0, case["vocab"])], tokens, s.pick.data_ptr(), stream)
        return logits, s.pick
    return [y for launch in s.launches for y in launch[2]]


def _exact_products(case, seed):
    out, part = [], 0
    for rows, columns in _case_products(case):
        x = _acts(case["tokens"], columns, seed + part)
        x = _int8_codes(x) if case["act"] == "int8" else x.to(F64)
        for r in rows:
            out.append(x @ _unpack(case["fmt"], _matrix(case["fmt"], r, columns, seed, part), columns).t())
            part += 1
    if case["kind"] == "host":
        return out[0].cpu().numpy()
    return (out[0], None) if case["kind"] == "head" else out


# ---- requests ---------------------------------------------------------------------------------------------------------------

STEP = 7      # the successor of token t is STEP * t + 3, modulo the vocabulary


def _successor(case, token):
    return (STEP * token + 3) % case["vocab"]


def _heads(case):
    w = case["width"]
    return dict(heads=w // 128, kv_heads=max(w // 256, 4) if w < 4096 else 8, dim=128)


def _prompt(case, seed):
    return torch.randint(0, case["vocab"], (case["prompt"],), generator=_generator(seed, 998), device=DEV).tolist()


def _positions(case):
    return case["prompt"] + case["new"]


def _llama_config(case):
    h = _heads(case)
    return LlamaConfig(embedding=case["width"], layers=case["layers"], heads=h["heads"], kv_heads=h["kv_heads"], head_dim=h["dim"], ffn=HIDDEN[case["width"]],
                       vocab=case["vocab"], context=_positions(case))


def _embedding(case, seed):
    return torch.randn((case["vocab"], case["width"]), generator=_generator(seed, 0), device=DEV)


def _head_rows(case, embedding):
    """The head's row of a token is the embedding of the token it follows."""
    before = (torch.arange(case["vocab"], device=DEV) - 3) * pow(STEP, -1, case["vocab"]) % case["vocab"]
    return embedding[before] * case["width"] ** -0.5


def _llama_tensors(case, seed):
    """(name, raw Q8_0 rows or fp32 vector on the device, is_matrix)"""
    for part, (name, shape, is_matrix) in enumerate(llama_plan(_llama_config(case))):
        if name == "token_embd.weight":
            yield name, _pack("Q8_0", _embedding(case, seed)), True
        elif name == "output.weight":
            yield name, _pack("Q8_0", _head_rows(case, _embedding(case, seed))), True
        elif is_matrix:
            yield name, _matrix("Q8_0", *shape, seed, part), True
        else:
            yield name, 1.0 + 0.1 * torch.randn(shape, generator=_generator(seed, part), device=DEV), False


def _kipirax_dict(case):
    h = _heads(case)
    H, G, D = h["heads"], h["kv_heads"], h["dim"]
    mixers = {"channel_delta": dict(heads=H, kv_heads=H, dim=D, vdim=D, conv=4),
              "parallel": dict(left=dict(heads=H, kv_heads=G, dim=D, vdim=D, scale=D ** -0.5, mask=dict(size=1024, keep_first=4)), right=dict(heads=H, dim=D, vdim=D))}
    return dict(architecture="Kipirax", width=case["width"], vocab=case["vocab"], max_positions=_positions(case), norm=dict(eps=1e-6, groups=4), logit_softcap=30.0,
                layers=[dict(type=kind, mixer=mixers[kind], mlp=dict(kind="dense", ff=HIDDEN[case["width"]])) for kind in
                        (("channel_delta", "parallel")[i % 2] for i in range(case["layers"]))])


def _sikivik_dict(case):
    h = _heads(case)
    H, G, D = h["heads"], h["kv_heads"], h["dim"]
    rot = dict(base=1e5, dims=D)
    window = dict(heads=H, kv_heads=G, dim=D, vdim=D, scale=D ** -0.5, mask=dict(size=1024), conv=4, rot=rot, v_mix=True)
    kinds = [("attention", window), ("retention", dict(heads=H, dim=D, vdim=D, rot=rot, decay=[1.0 - 2.0 ** (-5.0 - 5.0 * i / H) for i in range(H)])),
             ("attention", window), ("gla", dict(heads=H, dim=D, vdim=D, tau=16.0))]
    return dict(architecture="Sikivik", width=case["width"], vocab=case["vocab"], norm=dict(eps=1e-6),
                layers=[dict(type=kinds[i % 4][0], mixer=kinds[i % 4][1], mlp=dict(kind="dense", ff=HIDDEN[case["width"]])) for i in range(case["layers"])])


def _dense_model(case):
    """(decoder class, configuration, [(name, shape)], the package's made-up small tensors)"""
    if case["arch"] == "kipirax":
        cfg, rank = KipiraxConfig.from_dict(_kipirax_dict(case)), 64 if case["width"] == 1024 else 128
        return KipiraxDecoder, cfg, kipirax_plan(cfg, rank, rank), kipirax_tensor
    cfg = SikivikConfig.from_dict(_sikivik_dict(case))
    return SikivikDecoder, cfg, sikivik_plan(cfg, 16), sikivik_tensor


def _dense_tensor(case, seed, plan, small):
    """name -> bfloat16 tensor on the device"""
    number = {name: (i + 1, shape) for i, (name, shape) in enumerate(plan)}

    def tensor(name):
        part, shape = number[name]
        if name == "embed":
            t = 2.0 * _embedding(case, seed)
        elif name == "head":
            t = _head_rows(case, _embedding(case, seed))
        elif len(shape) == 2 and shape[0] * shape[1] > 1 << 16:
            t = torch.randn(shape, generator=_generator(seed, part), device=DEV) * (0.5 if name == "pos" else shape[1] ** -0.5)
        else:
            t = torch.from_numpy(np.asarray(small(name, shape, np.random.default_rng([seed, part])))).to(DEV)
        return t.to(torch.bfloat16)
    return tensor


def _prepare_request(case, seed):
    s = Held(case)
    s.prompt = _prompt(case, seed)
    if case["arch"] == "llama":
        tensors = ((name, t.cpu().numpy(), is_matrix) for name, t, is_matrix in _llama_tensors(case, seed))
        s.decoder = LlamaDecoder(_backend(), _llama_config(case), tensors, act_mode=MODES[case["act"]])
    else:
        decoder, cfg, plan, small = _dense_model(case)
        device = _dense_tensor(case, seed, plan, small)
        s.decoder = decoder(_backend(), cfg, lambda name: device(name).view(torch.int16).cpu().numpy().view(np.uint16), max_positions=_positions(case))
    s.decoder.capture()
    return s


def _run_request(s):
    d = s.decoder
    tokens = d.generate(s.prompt, s.case["new"])
    return torch.tensor(tokens), d.logits


# ---- what a request's last logits are in 64 bits ------------------------------------------------------------------------------

def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _silu(x):
    return x * torch.sigmoid(x)


def _softmax_attention(q, k, v, scale, seen, bias=None):
    """q [T, H, D], k, v [T, G, .]; seen [T, T]; bias [H] times the distance"""
    T, H = q.shape[:2]
    of = torch.arange(H, device=DEV) // (H // k.shape[1])
    s = torch.einsum("ihd,jhd->hij", q, k[:, of]) * scale
    if bias is not None:
        at = torch.arange(T, device=DEV, dtype=F64)
        s = s - bias[:, None, None] * (at[:, None] - at[None, :])
    p = torch.softmax(s.masked_fill(~seen, -math.inf), -1)
    return torch.einsum("hij,jhd->ihd", p, v[:, of])


def _window(T, size, keep_first=0):
    at = torch.arange(T, device=DEV)
    back = at[:, None] - at[None, :]
    return (back >= 0) & ((back < size) | (at[None, :] < keep_first))


def _conv(x, taps):
    """x [T, C], taps [C, n]: causal, per channel"""
    n = taps.shape[1]
    x = torch.cat([torch.zeros((n - 1, x.shape[1]), dtype=F64, device=DEV), x])
    T = x.shape[0] - n + 1
    return sum(x[j:j + T] * taps[:, j] for j in range(n))


def _matrix_states(q, k, v, g, beta=None):
    """S <- g S (+ the delta rule's correction), S <- S + k u^T, o = S^T q; all [T, H, .]"""
    S = torch.zeros((q.shape[1], k.shape[2], v.shape[2]), dtype=F64, device=DEV)
    out = torch.empty_like(v)
    for t in range(q.shape[0]):
        S = S * g[t][:, :, None]
        u = v[t] if beta is None else beta[t][:, None] * (v[t] - torch.einsum("hdv,hd->hv", S, k[t]))
        S = S + k[t][:, :, None] * u[:, None, :]
        out[t] = torch.einsum("hdv,hd->hv", S, q[t])
    return out


def _rotate_half(x, base):
    T, _, D = x.shape
    angle = torch.arange(T, device=DEV, dtype=F64)[:, None] * base ** (-torch.arange(0, D, 2, device=DEV, dtype=F64) / D)
    c, s = torch.cos(angle)[:, None], torch.sin(angle)[:, None]
    a, b = x[..., :D // 2], x[..., D // 2:]
    return torch.cat([a * c - b * s, b * c + a * s], -1)


def _llama_logits(case, seed, tokens):
    cfg = _llama_config(case)
    H, G, D, T = cfg.heads, cfg.kv_heads, cfg.head_dim, len(tokens)
    given = _int8_codes if case["act"] == "int8" else lambda x: x
    i = torch.arange(D // 2, device=DEV, dtype=torch.float32)
    angle = (torch.arange(T, device=DEV, dtype=torch.float32)[:, None] * torch.pow(cfg.rope_base, -2.0 * i / D)).to(F64)      # the model's tables are of 32-bit angles
    c, s = torch.cos(angle)[:, None], torch.sin(angle)[:, None]

    def turn(x):
        a, b = x[..., 0::2], x[..., 1::2]
        return torch.stack([a * c - b * s, a * s + b * c], -1).flatten(-2)

    raw = {name: t for name, t, _ in _llama_tensors(case, seed)}
    mul = lambda x, name: given(x) @ _unpack("Q8_0", raw[name], x.shape[-1]).t()
    norm = lambda x, name: _rms(x, cfg.rms_eps) * raw[name].to(F64)
    x = _unpack("Q8_0", raw["token_embd.weight"][torch.tensor(tokens, device=DEV)].contiguous(), cfg.embedding)
    seen = _window(T, T)
    for layer in range(cfg.layers):
        p = f"blk.{layer}."
        h = norm(x, p + "attn_norm.weight")
        q, k, v = (mul(h, f"{p}attn_{n}.weight").view(T, -1, D) for n in "qkv")
        x = x + mul(_softmax_attention(turn(q), turn(k), v, D ** -0.5, seen).reshape(T, H * D), p + "attn_output.weight")
        h = norm(x, p + "ffn_norm.weight")
        x = x + mul(_silu(mul(h, p + "ffn_gate.weight")) * mul(h, p + "ffn_up.weight"), p + "ffn_down.weight")
    return mul(norm(x[-1:], "output_norm.weight"), "output.weight")[0]


def _kipirax_logits(c, w, tokens):
    eps, groups, T = c["norm"]["eps"], c["norm"]["groups"], len(tokens)
    grouped = lambda x, weight: _rms(x.view(T, groups, -1), eps).reshape(T, -1) * weight
    x = w("embed")[torch.tensor(tokens, device=DEV)] + w("pos")[:T]
    for i, layer in enumerate(c["layers"]):
        p, m = f"l{i}.", layer["mixer"]
        mix = lambda n: w(p + "mix." + n)
        h = x + (torch.cat([torch.zeros_like(x[:1]), x[:-1]]) - x) * w(p + "shift")
        if layer["type"] == "channel_delta":
            H, D = m["heads"], m["dim"]
            q, k, v = (_silu(_conv(h @ mix(n).t(), mix(n + ".conv"))).view(T, H, -1) for n in "qkv")
            unit = lambda z: z / torch.sqrt((z * z).sum(-1, keepdim=True) + 1e-6)
            rate = torch.nn.functional.softplus(h @ mix("a1").t() @ mix("a2").t() + mix("dt_bias"), threshold=100.0).view(T, H, D)
            o = _matrix_states(unit(q) * D ** -0.5, unit(k), v, torch.exp(-torch.exp(mix("A_log"))[:, None] * rate), torch.sigmoid(h @ mix("b").t()))
            y = ((_rms(o, eps) * mix("norm")).reshape(T, -1) * torch.sigmoid(h @ mix("g1").t() @ mix("g2").t())) @ mix("o").t()
        else:
            a, r = m["left"], m["right"]
            H, G, D = a["heads"], a["kv_heads"], a["dim"]
            q, k = (_rms((h @ mix(f"left.{n}").t()).view(T, -1, D), eps) * mix(f"left.{n}.norm") for n in "qk")
            bias = 2.0 ** (-8.0 * torch.arange(1, H + 1, device=DEV, dtype=F64) / H)
            o = _softmax_attention(q, k, (h @ mix("left.v").t()).view(T, G, -1), a["scale"], _window(T, a["mask"]["size"], a["mask"]["keep_first"]), bias)
            left = (o * torch.sigmoid(h @ mix("left.g").t())[:, :, None]).reshape(T, -1) @ mix("left.o").t()
            H, D = r["heads"], r["dim"]
            f = mix("right.lower") + (1.0 - mix("right.lower")) * torch.sigmoid(h @ mix("right.f").t() + mix("right.f.b"))
            f = f.view(T, H, D)
            o = _matrix_states(_silu(h @ mix("right.q").t()).view(T, H, D), 1.0 - f, (h @ mix("right.v").t()).view(T, H, -1), f)
            right = (_rms(o, eps) * mix("right.norm")).reshape(T, -1) @ mix("right.o").t()
            y = 0.5 * (_rms(left, eps) * mix("left.out") + _rms(right, eps) * mix("right.out"))
        x = x + grouped(y, w(p + "norm1"))
        x = x + grouped(torch.relu(x @ w(p + "mlp.up").t()) ** 2 @ w(p + "mlp.down").t(), w(p + "norm2"))
    logits = grouped(x, w("final.norm"))[-1] @ w("head").t()
    return c["logit_softcap"] * torch.tanh(logits / c["logit_softcap"])


def _sikivik_logits(c, w, tokens):
    eps, T, first = c["norm"]["eps"], len(tokens), None
    x = w("embed")[torch.tensor(tokens, device=DEV)]
    for i, layer in enumerate(c["layers"]):
        p, m = f"l{i}.", layer["mixer"]
        mix = lambda n: w(p + "mix." + n)
        H, D = m["heads"], m["dim"]
        h = _rms(x, eps) * w(p + "norm1")
        if layer["type"] == "attention":
            G = m["kv_heads"]
            q, k, v = (_conv(h @ mix(n).t() + mix(n + ".b"), mix(n + ".conv")) for n in "qkv")
            q, k, v = _rotate_half(q.view(T, H, D), m["rot"]["base"]), _rotate_half(k.view(T, G, D), m["rot"]["base"]), v.view(T, G, -1)
            v = v if first is None else (1.0 - mix("vmix")) * v + mix("vmix") * first
            first = v if first is None else first
            o = _softmax_attention(q, k, v, m["scale"], _window(T, m["mask"]["size"]))
            y = (o.reshape(T, -1) * torch.sigmoid(h @ mix("g").t())) @ mix("o").t() + mix("o.b")
        else:
            q, k, v = ((h @ mix(n).t()).view(T, H, -1) for n in "qkv")
            if layer["type"] == "gla":
                q = q * D ** -0.5
                decay = torch.exp(torch.nn.functional.logsigmoid(h @ mix("a1").t() @ mix("a2").t() + mix("a2.b")) / m["tau"]).view(T, H, D)
                o = _rms(_matrix_states(q, k, v, decay), eps) * mix("norm")
            else:
                q, k = _rotate_half(q, m["rot"]["base"]), _rotate_half(k, m["rot"]["base"]) * D ** -0.5
                decay = torch.tensor(m["decay"], device=DEV, dtype=F64)[None, :, None].expand(T, H, D)
                o = _rms(_matrix_states(q, k, v, decay), eps)
            y = (o.reshape(T, -1) * _silu(h @ mix("g").t())) @ mix("o").t()
        x = x + y + (_silu(h @ w(p + "mlp.gate").t()) * (h @ w(p + "mlp.up").t())) @ w(p + "mlp.down").t()
    return (_rms(x[-1:], eps) * w("final.norm"))[0] @ w("head").t()


def _exact_request(case, seed):
    tokens = _prompt(case, seed)
    for _ in range(case["new"] - 1):
        tokens.append(_successor(case, tokens[-1]))
    if case["arch"] == "llama":
        return None, _llama_logits(case, seed, tokens)
    _, _, plan, small = _dense_model(case)
    tensor = _dense_tensor(case, seed, plan, small)
    w = lambda name: tensor(name).to(F64)
    return None, (_kipirax_logits(_kipirax_dict(case), w, tokens) if case["arch"] == "kipirax" else _sikivik_logits(_sikivik_dict(case), w, tokens))


# ---- the interface ----------------------------------------------------------------------------------------------------------

def prepare(case, seed):
    return _prepare_request(case, seed) if case["kind"] == "request" else _prepare_products(case, seed)


def run(state):
    return _run_request(state) if state.case["kind"] == "request" else _run_products(state)


def exact(case, seed):
    return _exact_request(case, seed) if case["kind"] == "request" else _exact_products(case, seed)


def work(case):
    if case["kind"] != "request":
        per, size = BLOCK[case["fmt"]]
        weights = sum(sum(rows) * columns for rows, columns in _case_products(case))
        vectors = sum(columns + sum(rows) for rows, columns in _case_products(case)) * case["tokens"] * 4
        return dict(bytes=weights * size // per + vectors, flops=2 * weights * case["tokens"])
    # a request: the weights once for the prompt and once for every further token, the caches as far as they are filled
    W, V, F = case["width"], case["vocab"], HIDDEN[case["width"]]
    h, prompt, steps = _heads(case), case["prompt"], case["new"] - 1
    H, G, D = h["heads"], h["kv_heads"], h["dim"]
    attention, state = H * D * 2 + G * D * 2, 0
    if case["arch"] == "llama":
        layer, item = W * attention + 3 * W * F, 34 / 32
        attends, layers = case["layers"], layer * case["layers"]
    elif case["arch"] == "sikivik":
        item, attends = 2, case["layers"] // 2
        layers = attends * (2 * 3 * W * F + W * (attention + H * D) + W * 5 * H * D)
        state = attends * H * D * D
    else:
        item, attends = 2, case["layers"] // 2
        layers = attends * (2 * 2 * W * F + W * 4 * H * D + W * (attention + 4 * H * D))
        state = 2 * attends * H * D * D
    window = 1 << 30 if case["arch"] == "llama" else 1024
    keys = sum(min(t + 1, window) for t in range(prompt + steps)) * attends          # (query, key) pairs of one head
    step_keys = sum(min(prompt + t + 1, window) for t in range(steps)) * attends
    nbytes = (layers * (1 + steps) + V * W * case["new"]) * item + (step_keys + min(prompt, window) * attends) * 2 * G * D * 4 + 8 * state * (1 + steps)
    flops = 2 * layers * (prompt + steps) + 2 * V * W * case["new"] + 4 * keys * H * D + 6 * state * (prompt + steps)
    return dict(bytes=nbytes, flops=flops)


def tolerance(case):
    """About four times what the paths show against 64 bits."""
    if case["kind"] == "request":
        # int8 activations: a code that rounds the other way moves everything behind it (1e-2); bf16: a prompt's products (8e-4)
        return {"rel": {"int8": 0.03, "bf16": 0.004, "fp32": 2.5e-4}[case["act"]], "differ": 0.005}
    if case["kind"] == "block" or case["tokens"] > 6:
        return {"rel": 2.5e-4}      # weights and activations in 16-bit fixed point per 256 (6e-5)
    if case["act"] == "int8":
        return {"rel": 1e-5}        # whole-number dot products, 32-bit sums of their scaled blocks (1e-7)
    return {"rel": 1e-4}            # activations in 16-bit fixed point per 32 (2e-5)
