"""What users of this library have the GPU do, as cases that can be timed and compared.

Four kinds of call:

  step       one segment of every stream through the model plugin, in the order an encoder makes the
             calls: forward pass, coder-ready values, backward pass, RMSProp update, memory shift, with
             ids and targets in host memory and the coder values and the loss back in host memory
  decode     the one-symbol steps of one segment: forward pass, coder trees and range decoder on the
             device, the decoded symbols back in host memory
  attention  the isolated attention op, forward and backward, on device tensors
  file       a short file compressed and decompressed, with the model made for each as the command line does

The states are those of a job in full run: the memory holds a segment and RMSProp's second moments
the size of the gradients (zero moments turn the first update into the gradient's sign, which
rounding decides for small gradients).
"""
import ctypes as C
import importlib.util
import math
import os
import sys

import numpy as np
import torch


def _package():
    """The package of the repository in the working folder (its folder's name is not an identifier)."""
    name = "nncp_metal_b200"
    if name not in sys.modules:
        folder = os.path.abspath("nncp-metal_b200")
        spec = importlib.util.spec_from_file_location(name, os.path.join(folder, "__init__.py"),
                                                      submodule_search_locations=[folder])
        sys.modules[name] = module = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(module)
    return sys.modules[name]


# ---------------------------------------------------------------- the cases

# ln_flags and ff_act as in include/nncu.h
_POST, _PRE_FINAL_RMS, _GELU, _GEGLU = 1, 2 | 4 | 16, 1, 2

_CONFIG0 = dict(n_layer=2, d_model=128, n_head=4, d_inner=512, seg_len=32, mem_len=32, d_pos=64, n_streams=4,
                n_symbols=256, bf16=0, tied=0, ln=_POST, act=_GELU)
_LEVEL6 = dict(n_layer=4, d_model=256, n_head=8, d_inner=512, seg_len=32, mem_len=32, d_pos=32, n_streams=16,
               n_symbols=256, bf16=0, tied=1, ln=_POST, act=_GELU)
_LEVEL9 = dict(_LEVEL6, n_layer=6, d_model=512, d_inner=1024, seg_len=64, mem_len=64, d_pos=64, bf16=1)
_CONFIG2 = dict(n_layer=12, d_model=512, n_head=8, d_inner=2048, seg_len=64, mem_len=64, d_pos=128, n_streams=32,
                n_symbols=16384, bf16=1, tied=0, ln=_POST, act=_GELU)
_CONFIG3 = dict(_CONFIG2, n_layer=20, d_model=1024, n_head=16, d_inner=4096, mem_len=256, d_pos=320, n_streams=64)
_CONFIG4 = dict(_CONFIG2, mem_len=512, d_pos=576, n_streams=128)
_ENWIK = dict(_CONFIG3, n_head=8, d_inner=3072, n_streams=32, ln=_PRE_FINAL_RMS, act=_GEGLU)
# text through the word tokenizer: an alphabet that is no power of two, streams and lengths that fill no tile
_WORDS = dict(_CONFIG2, n_layer=8, seg_len=50, mem_len=77, d_pos=100, n_streams=13, n_symbols=9208, ln=_PRE_FINAL_RMS,
              act=_GEGLU)


def listed():
    return [
        # the smallest model that is in use: bytes, fp32; a step is launches and host calls
        dict(name="step config0", kind="step", **_CONFIG0),
        # levels 4-6 (default) and 7-9 of the command line
        dict(name="step level6", kind="step", **_LEVEL6),
        dict(name="step level9", kind="step", **_LEVEL9),
        # the text model the headline figure is quoted on
        dict(name="step config2", kind="step", **_CONFIG2),
        # tokenised text with a ragged shape
        dict(name="step words", kind="step", **_WORDS),
        # the large models: wide heads and gated activations; deep and wide; long memory and many streams
        dict(name="step enwik", kind="step", **_ENWIK),
        dict(name="step config3", kind="step", **_CONFIG3),
        dict(name="step config4", kind="step", **_CONFIG4),
        # decoding: the default level's small model, and many streams over a long memory
        dict(name="decode level6", kind="decode", **_LEVEL6),
        dict(name="decode config4", kind="decode", **_CONFIG4),
        # the attention op by itself: 16 streams, 8 heads of 64, 64 queries over 64 + 64 keys
        dict(name="attention config1", kind="attention", n_streams=16, n_head=8, d_key=64, seg_len=64, mem_len=64,
             d_pos=128, bf16=1),
        # a short file at the default level, there and back
        dict(name="file level6", kind="file", n_bytes=12000, **_LEVEL6),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_model(rng):
    if rng.random() < 0.25:  # the fp32 models of the lower levels
        heads = rng.randint(2, 8)
        c = dict(n_layer=rng.randint(2, 4), n_head=heads, d_model=32 * heads, d_inner=64 * heads * rng.randint(1, 2),
                 seg_len=rng.randint(16, 32), mem_len=rng.randint(8, 40), n_streams=_log_int(rng, 1, 16), n_symbols=256,
                 bf16=0, tied=rng.randint(0, 1), ln=_POST, act=_GELU)
    else:
        d_key = rng.choice((32, 64, 64, 64, 128))
        heads = _log_int(rng, max(2, 256 // d_key), 1024 // d_key)
        big_alphabet = rng.random() < 0.7
        # byte alphabets and dictionaries: every size a multiple of 8, half of them powers of two
        symbols = _log_int(rng, 1024, 16384) // 8 * 8 if big_alphabet else 256
        if rng.random() < 0.5:
            symbols = 1 << int(math.log2(symbols))
        c = dict(n_layer=_log_int(rng, 2, 20), n_head=heads, d_model=d_key * heads,
                 d_inner=d_key * heads * rng.randint(2, 4), seg_len=rng.choice((64, 64, rng.randint(16, 64))),
                 mem_len=_log_int(rng, 16, 512), n_streams=_log_int(rng, 1, 128), n_symbols=symbols, bf16=1,
                 tied=rng.randint(0, 1), ln=rng.choice((_POST, _PRE_FINAL_RMS)), act=rng.choice((_GELU, _GEGLU)))
    keys = c["seg_len"] + c["mem_len"]
    c["d_pos"] = rng.choice((keys, rng.randint(keys // 2, keys)))
    return c


def draw(rng):
    kind = rng.choice(("step",) * 11 + ("decode",) * 4 + ("attention",) * 4 + ("file",))
    if kind == "attention":
        c = dict(kind=kind, n_streams=_log_int(rng, 1, 128), n_head=_log_int(rng, 4, 16), d_key=rng.choice((32, 64, 64, 128)),
                 seg_len=rng.choice((64, rng.randint(16, 64))), mem_len=_log_int(rng, 16, 512), bf16=1)
        if rng.random() < 0.2:
            c.update(d_key=32, seg_len=rng.randint(16, 32), mem_len=rng.randint(8, 40), bf16=0)
        keys = c["seg_len"] + c["mem_len"]
        c["d_pos"] = rng.choice((keys, rng.randint(keys // 2, keys)))
        return c
    if kind == "file":
        return dict(_LEVEL6, kind=kind, n_layer=rng.randint(2, 4), n_streams=_log_int(rng, 4, 16),
                    n_bytes=_log_int(rng, 2000, 12000))
    most = 1e13 if kind == "step" else 2.6e12  # the work of the largest listed case of the kind
    while True:
        c = dict(_draw_model(rng), kind=kind)
        if work(c)["flops"] <= most:
            return c


# ---------------------------------------------------------------- inputs

def _tokens(rng, n_streams, length, n_symbols):
    """[length][n_streams] symbols: a Zipf(1.1) unigram mixed half and half with an order-1 Markov chain."""
    zipf = np.arange(1, n_symbols + 1) ** -1.1
    drawn = np.searchsorted(np.cumsum(zipf / zipf.sum()), rng.random((length, n_streams))).clip(0, n_symbols - 1)
    successor = rng.integers(0, min(n_symbols, 512), size=(n_symbols, 8))
    pick = rng.integers(0, 8, (length, n_streams))
    fresh = rng.random((length, n_streams)) < 0.5
    out = np.zeros((length, n_streams), np.int32)
    last = np.zeros(n_streams, np.int32)
    for t in range(length):
        last = np.where(fresh[t], drawn[t], successor[last, pick[t]])
        out[t] = last
    return out


def _params(c, seed):
    return _package().abi.make_params(
        n_layer=c["n_layer"], d_model=c["d_model"], n_head=c["n_head"], d_key=c["d_model"] // c["n_head"],
        d_inner=c["d_inner"], d_pos=c["d_pos"], mem_len=c["mem_len"], seg_len=c["seg_len"], n_streams=c["n_streams"],
        n_symbols=c["n_symbols"], use_bf16=c["bf16"], tied_w_r=c["tied"], tied_b_r=c["tied"], query_bias=1,
        ln_flags=c["ln"], ff_act=c["act"], init_kind=_package().abi.INIT_UNIFORM, init_range=0.035 * c["d_model"] ** 0.5,
        seed=seed & 0x7FFFFFFF, lr=3e-4, beta2=0.99, eps=1e-8)


SEGMENTS = 4


def _ptr(a):
    return a.ctypes.data_as(C.c_void_p)


def _view(m, pointer, n):
    """One of the model's device buffers as a tensor that keeps the model alive."""
    array = _package().dist.CudaArray(pointer, n)
    array.model = m
    return torch.as_tensor(array, device="cuda")


def _model(c, seed, tokens):
    """A model in full run on a stream of its own: one segment in memory, second moments of the gradients' size."""
    m = _package().TrfModel(_params(c, seed))
    stream = torch.cuda.Stream()
    m.set_stream(stream.cuda_stream)
    m.reset()
    T = c["seg_len"]
    m.eval(-1, tokens[:T], read=False)
    m.eval_gradient(tokens[1:T + 1])
    m.memory_shift()
    m.synchronize()
    w, g, v, n = m.flat_buffers()
    flat = {k: _view(m, p, n) for k, p in (("weights", w), ("grads", g), ("moments", v))}
    for at, count in m.info.values():
        flat["moments"][at:at + count] = flat["grads"][at:at + count].square().mean() + 1e-18
    torch.cuda.synchronize()
    return m, stream, flat


def _prepare_step(c, seed):
    T, B, V = c["seg_len"], c["n_streams"], c["n_symbols"]
    tokens = _tokens(np.random.default_rng(seed), B, (SEGMENTS + 1) * T + 1, V)
    m, stream, flat = _model(c, seed, tokens)
    cut = [(np.ascontiguousarray(tokens[k * T:(k + 1) * T]), np.ascontiguousarray(tokens[k * T + 1:(k + 1) * T + 1]))
           for k in range(1, SEGMENTS + 1)]
    probs = _view(m, m.probs_dev(), T * B * V)
    bits = (V - 1).bit_length()
    return dict(kind="step", m=m, stream=stream, outputs=dict(flat, probs=probs), segments=cut, at=0, lr=3e-4,
                paths=np.zeros((T * B, bits), np.uint16), n_bits=C.c_int())


def _run_step(s):
    m = s["m"]
    ids, targets = s["segments"][s["at"] % SEGMENTS]
    s["at"] += 1
    m.eval(-1, ids, read=False)
    m._ck(m.lib.nncu_coder_paths_begin(m.h, 0, m.T, _ptr(targets)))
    m.set_lr(s["lr"])
    m._ck(m.lib.nncu_eval_gradient(m.h, _ptr(targets), None))
    m.update()
    m._ck(m.lib.nncu_coder_paths_end(m.h, _ptr(s["paths"]), C.byref(s["n_bits"])))
    # the coder's 15-bit integers as the probabilities they stand for: their last bits follow the model's rounding
    return dict(s["outputs"], prob0=s["paths"].astype(np.float32), loss=m.read_loss())


def _prepare_decode(c, seed):
    host = _package().host
    T, B, V = c["seg_len"], c["n_streams"], c["n_symbols"]
    tokens = _tokens(np.random.default_rng(seed), B, 2 * T + 1, V)
    m, stream, _ = _model(c, seed, tokens)
    targets = np.ascontiguousarray(tokens[T + 1:2 * T + 1])
    m.eval(-1, tokens[T:2 * T], read=False)
    paths = m.coder_paths(0, T, targets)
    m.eval_end()
    lib = host.library()
    enc, data = lib.nch_enc_new(), C.c_void_p()
    lib.nch_write_sym_paths_any(enc, _ptr(paths), V, _ptr(targets), T * B)
    n = lib.nch_enc_finish(enc, C.byref(data))
    payload = C.string_at(data.value, n)
    lib.nch_enc_free(enc)
    return dict(kind="decode", m=m, stream=stream, payload=payload, ids=np.ascontiguousarray(tokens[T]))


def _run_decode(s):
    m = s["m"]
    m.decoder_begin(s["payload"])
    symbols = m.decode_steps(0, m.T, s["ids"])
    m.eval_end()
    m.decoder_end()
    return symbols


def _prepare_attention(c, seed):
    B, H, dk, T, M, P = (c[k] for k in ("n_streams", "n_head", "d_key", "seg_len", "mem_len", "d_pos"))
    L, HD = M + T, H * dk
    g = torch.Generator(device="cuda").manual_seed(seed)
    kind = torch.bfloat16 if c["bf16"] else torch.float32

    def normal(*shape, scale=1.0, dtype=kind):
        return (scale * torch.randn(*shape, generator=g, device="cuda")).to(dtype)

    q, kv, dout = normal(T * B, HD), normal(L * B, 2 * HD), normal(T * B, HD)
    w_r, b_r = normal(H, P, dk, scale=0.02, dtype=torch.float32), normal(H, L, scale=0.02, dtype=torch.float32)
    new = {"out": torch.zeros_like(q), "lse": torch.zeros(B * H, T, device="cuda"), "dq": torch.zeros_like(q),
           "dkv": torch.zeros_like(kv), "dw_r": torch.zeros_like(w_r), "db_r": torch.zeros_like(b_r)}
    parts = torch.zeros(B, H, P, dk, device="cuda"), torch.zeros(B, H, L, device="cuda")
    shape = _package().abi.AttnShape(B, H, dk, T, M, P, 0, 0, T, float(math.sqrt(dk * 512.0)), c["bf16"])
    return dict(kind="attention", lib=_package().library(), shape=shape, tensors=(q, kv, w_r, b_r, dout), new=new, parts=parts)


def _run_attention(s):
    lib, shape, new = s["lib"], C.byref(s["shape"]), s["new"]
    q, kv, w_r, b_r, dout = (t.data_ptr() for t in s["tensors"])
    out, lse, dq, dkv, dw_r, db_r = (new[k].data_ptr() for k in ("out", "lse", "dq", "dkv", "dw_r", "db_r"))
    dwr_part, dbr_part = (t.data_ptr() for t in s["parts"])
    st = torch.cuda.current_stream().cuda_stream
    if (lib.nncu_attention_forward(shape, q, kv, w_r, b_r, out, lse, st) or
            lib.nncu_attention_backward(shape, q, kv, w_r, b_r, out, lse, dout, dq, dkv, dwr_part, dbr_part, st) or
            lib.nncu_attention_reduce_tables(shape, dwr_part, dbr_part, dw_r, db_r, 0, st)):
        raise RuntimeError(lib.nncu_last_error().decode())
    return new


def _prepare_file(c, seed):
    rng = np.random.default_rng(seed)
    return dict(kind="file", params=_params(c, seed), symbols=_tokens(rng, 1, c["n_bytes"], c["n_symbols"])[:, 0].astype(np.uint16))


def _run_file(s):
    host = _package().host
    ops = host.bind_cuda(s["params"])
    data, _ = host.compress(ops, host.file_params(s["params"]), s["symbols"], host.EVAL_SEGMENT, host.OUT_CODER_READY)
    host.unbind_cuda(ops)
    ops = host.bind_cuda(s["params"])
    back = host.decompress(ops, data, host.OUT_DEVICE)
    host.unbind_cuda(ops)
    # the file's bytes follow the last bits of the model's sums, and a file is read by the build that wrote it:
    # what has to hold is that the symbols come back and that the file is as small
    return {"symbols": back, "file_bytes": float(len(data))}


_PREPARE = {"step": _prepare_step, "decode": _prepare_decode, "attention": _prepare_attention, "file": _prepare_file}
_RUN = {"step": _run_step, "decode": _run_decode, "attention": _run_attention, "file": _run_file}


def prepare(case, seed):
    return _PREPARE[case["kind"]](case, seed)


def run(state):
    return _RUN[state["kind"]](state)


# ---------------------------------------------------------------- what a pass cannot do without

def _attention_flops(c, heads_dim):
    """One contraction family: every query of every stream against `keys` rows of a head-wide operand."""
    return 2 * c["n_streams"] * c["seg_len"] * heads_dim


def _forward_flops(c):
    """(all contractions of the forward pass, those into the memory rows)"""
    D, F, T, M, B, V = (c[k] for k in ("d_model", "d_inner", "seg_len", "mem_len", "n_streams", "n_symbols"))
    up = 2 * F if c["act"] == _GEGLU else F
    memory = 2 * B * M * D * 2 * D
    layer = 2 * B * T * D * (4 * D + up + F) + memory + _attention_flops(c, D) * (2 * (M + T) + c["d_pos"])
    return c["n_layer"] * layer + 2 * B * T * D * V, c["n_layer"] * memory


def _n_params(c):
    D, F, V, L = c["d_model"], c["d_inner"], c["n_symbols"], c["mem_len"] + c["seg_len"]
    up = 2 * F if c["act"] == _GEGLU else F
    tables = c["d_pos"] * D + c["n_head"] * L
    return c["n_layer"] * (4 * D * D + (up + F) * D) + tables * (1 if c["tied"] else c["n_layer"]) + 2 * V * D


def work(case):
    c, kind = case, case["kind"]
    if kind == "attention":
        B, T, L, HD, e = c["n_streams"], c["seg_len"], c["seg_len"] + c["mem_len"], c["n_head"] * c["d_key"], 2 if c["bf16"] else 4
        # forward: scores, positions, values; backward: those two scores again and six gradients
        flops = _attention_flops(c, HD) * (2 * L + c["d_pos"] + 5 * L + 3 * c["d_pos"])
        tables = 4 * (c["n_head"] * L + HD * c["d_pos"])
        return {"bytes": e * B * HD * (4 * T + 4 * L) + 2 * tables, "flops": flops}
    T, B, V, D, e = c["seg_len"], c["n_streams"], c["n_symbols"], c["d_model"], 2 if c["bf16"] else 4
    n, (forward, memory) = _n_params(c), _forward_flops(c)
    # weights and moments in and out, gradients out; the probability table; the memory in and out
    step = {"bytes": 20 * n + 4 * T * B * V + 2 * e * c["n_layer"] * c["mem_len"] * B * D,
            "flops": 3 * forward - memory}
    # every symbol step needs the weights, the keys and values so far and a row of the table per stream
    decode = {"bytes": T * (e * (n - V * D) + c["n_layer"] * B * (c["mem_len"] + T // 2) * 2 * D * e + 12 * B * V), "flops": forward}
    if kind == "step":
        return step
    if kind == "decode":
        return decode
    segments = c["n_bytes"] / (T * B)
    return {k: 2 * segments * step[k] + segments * decode[k] for k in step}


def tolerance(case):
    if case["kind"] == "decode":
        return "exact"
    if case["kind"] == "file":
        return {"rel": 1e-3, "max": 1e-3, "differ": 0.0}
    # bf16: gradients whose terms cancel keep the rounding of the terms, so single small ones differ by more
    return {"rel": 1e-2, "max": 0.8} if case["bf16"] else {"rel": 3e-5, "max": 3e-3}
