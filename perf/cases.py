"""The work that programs have this library do, as cases to be timed.

A case is a dict: its `op` says which calls one pass makes, the other keys give sizes, widths, encodings and
source types.  M lhs rows, K depth, N rhs rows; (wa, ea) and (wb, eb) are the bits and the encoding of the two
operands ('u' unsigned, 's' signed, 'b' bipolar {-1, +1}).

  call     both operands imported from device memory, then the GEMM (the README's sequence)
  layer    one quantised layer at inference: the weights stay packed, the activations are imported (plainly, or
           against thresholds, `thr` of them per row), then the GEMM; `act` names the side of the activations
  forward  the GEMM alone, both operands packed
  host     the call with its operands and its result in pinned host memory
  train    one quantisation-aware training step: both operands imported, the GEMM, both gradients
  chain    the GEMMs of one network as a group: grouped import of new tensors, grouped GEMM
  group    a mix of GEMMs as a group captured with its imports, replayed
"""
from __future__ import annotations

import ctypes as C
import math

import torch

from gemmbitserial_gb300 import _capi, datagen
from gemmbitserial_gb300.api import allocGEMMContext, deallocGEMMContext, gemmBitSerial
from gemmbitserial_gb300.grouped import Group

_DTYPES = {"int8": torch.int8, "uint8": torch.uint8, "int16": torch.int16, "int32": torch.int32,
           "float32": torch.float32}


def _case(name, op, M, K, N, wa, ea, wb, eb, src="int8", act="rhs", col=False, thr=0):
    return {"name": name, "op": op, "M": M, "K": K, "N": N, "wa": wa, "ea": ea, "wb": wb, "eb": eb, "src": src,
            "act": act, "col": col, "thr": thr}


def listed():
    return [
        # the reference README's own example, the whole call: latency and launches
        _case("call_8x8192x8_u1u1", "call", 8, 8192, 8, 1, "u", 1, "u"),
        # CaffeNet's first fully connected layer, one sample: a matrix-vector product over 9 MB of weights
        _case("fc_4096x9216x1_u2u2", "layer", 4096, 9216, 1, 2, "u", 2, "u", "uint8"),
        # a CaffeNet convolution as a GEMM; its im2col buffer is feature-major, so it is read column-major
        _case("conv_384x2304x169_u2u2_col", "layer", 384, 2304, 169, 2, "u", 2, "u", "int8", "rhs", True),
        # the binary-net layer: a batch of bipolar activations against 4-bit signed weights
        _case("bnn_256x9216x4096_bps4", "layer", 256, 9216, 4096, 1, "b", 4, "s", "int8", "lhs"),
        # a layer fed by the int32 accumulators of the layer before it, requantised to 3 bits by 7 thresholds
        _case("requant_2048x4096x2048_s2u3", "layer", 2048, 4096, 2048, 2, "s", 3, "u", "int32", "rhs", False, 7),
        # 8-bit x 8-bit, the widest operands
        _case("int8_2048x4096x2048_s8s8", "layer", 2048, 4096, 2048, 8, "s", 8, "s"),
        # the headline GEMM, operands packed
        _case("forward_2048x4096x2048_u3s2", "forward", 2048, 4096, 2048, 3, "u", 2, "s"),
        # the headline GEMM as a program with host arrays calls it
        _case("host_2048x4096x2048_u3s2", "host", 2048, 4096, 2048, 3, "u", 2, "s"),
        # training steps, float inputs: a small layer of ragged sizes, and the named MLP layer
        _case("train_500x777x333_s4s4", "train", 500, 777, 333, 4, "s", 4, "s", "float32"),
        _case("train_4096x2048x2048_u2bp", "train", 4096, 2048, 2048, 2, "u", 1, "b", "float32"),
        # the CaffeNet chain: 8 GEMMs, odd and skinny ones among them, from newly made tensors
        {"name": "caffenet_chain", "op": "chain", "count": 0, "mix": 0},
        # the 512 uneven GEMMs of a quantised network in one graph: the largest call
        {"name": "group_512", "op": "group", "count": 512, "mix": datagen.SEED_BASE + 4},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    op = rng.choice(["call", "layer", "layer", "layer", "forward", "host", "train", "chain", "group"])
    if op == "chain" or op == "group":
        return {"op": op, "count": size(4, 64), "mix": rng.randrange(1 << 40)}
    even = rng.random() < 0.4  # whole multiples, as most layers have them; odd sizes otherwise

    def dims():
        m, k, n = size(1, 4096), size(64, 16384), size(1, 4096)
        return (m, k, n) if not even else (max(16, m // 16 * 16), k // 64 * 64, max(16, n // 16 * 16))

    M, K, N = dims()
    while M * K * N > 2048 * 4096 * 2048:
        M, K, N = dims()

    def enc():
        e = rng.choice("usb")
        if e == "b":
            return 1, e
        return (rng.randint(5, 8) if rng.random() < 0.15 else rng.randint(2 if e == "s" else 1, 4)), e

    (wa, ea), (wb, eb) = enc(), enc()
    src, act, col, thr = "int8" if max(wa, wb) < 8 else "int16", "rhs", False, 0
    if op == "train":
        src = "float32"
    elif op == "layer":
        act, col = rng.choice(["lhs", "rhs"]), rng.random() < 0.25
        if rng.random() < 0.3:
            bits = rng.randint(1, 4)
            src, thr = rng.choice(["int32", "float32"]), (1 << bits) - 1
            if act == "lhs":
                wa, ea = bits, "u"
            else:
                wb, eb = bits, "u"
        elif rng.random() < 0.5:
            src = rng.choice(["int16", "int32", "float32"])
    c = _case("", op, M, K, N, wa, ea, wb, eb, src, act, col, thr)
    del c["name"]
    return c


# ---------------------------------------------------------------- inputs

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) & 0x7FFFFFFFFFFFFFFF)
    return g


def _values(g, rows, cols, bits, enc, dtype=torch.int8):
    lo, hi = {"u": (0, (1 << bits) - 1), "s": (-(1 << (bits - 1)), (1 << (bits - 1)) - 1), "b": (0, 1)}[enc]
    v = torch.randint(lo, hi + 1, (rows, cols), generator=g, device="cuda", dtype=torch.int16)
    if enc == "b":
        v = v * 2 - 1
    return v.to(dtype)


def _mix(case):
    """The group's problems: (M, K, N, wA, encA, wB, encB)."""
    if case["op"] == "chain" and not case["count"]:
        return datagen.caffenet_mix()
    return datagen.grouped_mix(seed=case["mix"], count=case["count"])


def _operand(g, case, side):
    """(source as the program holds it, thresholds or None, the values the planes will encode)."""
    rows, bits, enc = (case["M"], case["wa"], case["ea"]) if side == "lhs" else (case["N"], case["wb"], case["eb"])
    K = case["K"]
    active = case["op"] != "layer" or case["act"] == side
    if active and case["thr"]:
        if case["src"] == "float32":
            x = torch.randn(rows, K, generator=g, device="cuda")
            t = torch.randn(case["thr"], rows, generator=g, device="cuda")
        else:  # accumulators of a layer before
            x = torch.randint(-3000, 3001, (rows, K), generator=g, device="cuda", dtype=torch.int32)
            t = torch.randint(-3000, 3001, (case["thr"], rows), generator=g, device="cuda", dtype=torch.int32)
        t = torch.sort(t, dim=0).values.contiguous()
        return x, t, lambda: torch.searchsorted(t.t().contiguous(), x).to(torch.int16)
    # weights (packed once) come as int8, 8-bit unsigned ones as int16
    dt = _DTYPES[case["src"]] if active else (torch.int16 if bits == 8 and enc == "u" else torch.int8)
    v = _values(g, rows, K, bits, enc, dt)
    return v, None, lambda: v


# ---------------------------------------------------------------- state

class _Contexts:
    """The contexts of a state and their group; frees them when nothing refers to them any more."""

    def __init__(self, ctxs):
        self.ctxs, self.group = ctxs, None

    def __del__(self):
        if self.group is not None:
            self.group.free()
        for c in self.ctxs:
            deallocGEMMContext(c)


class _State:
    """What a program holds between calls."""


class _DeviceArray:
    """A context's device result under the CUDA array interface; a tensor made of it keeps the contexts."""

    def __init__(self, owner, ptr, shape):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": "<i4", "version": 3}


def _import(side, x, thr, col):
    if thr is not None:
        side.importRegularAndQuantize(x, thr, readColMajor=col)
    else:
        side.importRegular(x, readColMajor=col)


def _prepare_group(case, seed):
    st, g, mix = _State(), _gen(seed), _mix(case)
    st.case = case
    st.src = [(datagen.torch_operand(g, M, K, wA, eA, "cuda"), datagen.torch_operand(g, N, K, wB, eB, "cuda"))
              for (M, K, N, wA, eA, wB, eB) in mix]
    st.lhs, st.rhs = [a for a, _ in st.src], [b for _, b in st.src]
    st.owner = _Contexts([allocGEMMContext(M, K, N, wA, wB, eA != "u", eB != "u")
                          for (M, K, N, wA, eA, wB, eB) in mix])
    st.owner.group = st.group = Group(st.owner.ctxs)
    st.views = [torch.as_tensor(_DeviceArray(st.owner, c.res_device, (N * M,)), device="cuda")
                for c, (M, K, N, *_) in zip(st.owner.ctxs, mix)]
    # a large group's results are handed on in one array
    st.flat = torch.empty(sum(v.numel() for v in st.views), dtype=torch.int32, device="cuda") if len(mix) > 64 else None
    torch.cuda.synchronize()
    if case["op"] == "group":
        s = torch.cuda.Stream()
        st.group.capture(st.lhs, st.rhs, stream=s)
        s.synchronize()
    return st


def prepare(case, seed):
    if case["op"] in ("chain", "group"):
        return _prepare_group(case, seed)
    st, g = _State(), _gen(seed)
    st.case = case
    M, K, N = case["M"], case["K"], case["N"]
    ctx = allocGEMMContext(M, K, N, case["wa"], case["wb"], case["ea"] != "u", case["eb"] != "u")
    st.owner, st.ctx = _Contexts([ctx]), ctx
    (a, ta, _), (b, tb, _) = _operand(g, case, "lhs"), _operand(g, case, "rhs")
    op = case["op"]
    st.out = torch.empty(N, M, dtype=torch.int32, device="cuda")
    if op == "host":
        a, b, st.out = a.cpu().pin_memory(), b.cpu().pin_memory(), torch.empty(N, M, dtype=torch.int32).pin_memory()
    elif op == "layer":
        x, t, w, side, wside = (a, ta, b, ctx.lhs, ctx.rhs) if case["act"] == "lhs" else (b, tb, a, ctx.rhs, ctx.lhs)
        wside.importRegular(w)
        st.x, st.t, st.side = (x.t().contiguous() if case["col"] else x), t, side
    elif op == "forward":
        ctx.lhs.importRegular(a)
        ctx.rhs.importRegular(b)
    elif op == "train":
        st.dC = torch.randn(N, M, generator=g, device="cuda")
        st.dA = torch.empty(M, K, device="cuda")
        st.dB = torch.empty(N, K, device="cuda")
    if op in ("call", "host", "train"):
        st.a, st.b = a, b
    torch.cuda.synchronize()
    return st


def run(st):
    op = st.case["op"]
    if op == "chain":
        st.group.import_(st.lhs, st.rhs)
        st.group.gemm()
    elif op == "group":
        st.group.replay()
    if op in ("chain", "group"):
        return st.views if st.flat is None else torch.cat(st.views, out=st.flat)
    ctx = st.ctx
    if op == "layer":
        _import(st.side, st.x, st.t, st.case["col"])
    elif op != "forward":
        ctx.lhs.importRegular(st.a)
        ctx.rhs.importRegular(st.b)
    gemmBitSerial(ctx, out=st.out)
    if op == "train":
        stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
        _capi.check(_capi.load().gbs_adjoint(ctx._h, C.c_void_p(st.dC.data_ptr()), C.c_void_p(st.dA.data_ptr()),
                                             C.c_void_p(st.dB.data_ptr()), stream))
        return {"res": st.out, "dA": st.dA, "dB": st.dB}
    return st.out


# ---------------------------------------------------------------- what a pass needs, and its exact results

def work(case):
    if case["op"] in ("chain", "group"):
        mix = _mix(case)
        return {"bytes": sum(M * K + N * K + 4 * M * N for (M, K, N, *_) in mix),
                "flops": sum(2.0 * M * K * N for (M, K, N, *_) in mix)}
    M, K, N, op = case["M"], case["K"], case["N"], case["op"]
    packed = {"lhs": case["wa"] * M * K / 8, "rhs": case["wb"] * N * K / 8}
    size = {"int8": 1, "uint8": 1, "int16": 2, "int32": 4, "float32": 4}[case["src"]]
    plain = {"lhs": size * M * K, "rhs": size * N * K}
    if op == "forward":
        operands = packed["lhs"] + packed["rhs"]
    elif op == "layer":
        other = "rhs" if case["act"] == "lhs" else "lhs"
        rows = M if case["act"] == "lhs" else N
        operands = plain[case["act"]] + 4 * case["thr"] * rows + packed[other]
    else:
        operands = plain["lhs"] + plain["rhs"]
    flops, nbytes = 2.0 * M * K * N, operands + 4 * M * N
    if op == "train":
        flops, nbytes = 3 * flops, nbytes + 4 * (M * N + M * K + N * K)
    return {"bytes": nbytes, "flops": flops}


def exact(case, seed):
    if work(case)["flops"] > 4e12:
        return None
    g = _gen(seed)
    if case["op"] in ("chain", "group"):
        ops = [(datagen.torch_operand(g, M, K, wA, eA, "cuda"), datagen.torch_operand(g, N, K, wB, eB, "cuda"))
               for (M, K, N, wA, eA, wB, eB) in _mix(case)]
        outs = [(b.double() @ a.double().t()).reshape(-1) for a, b in ops]
        return outs if len(outs) <= 64 else torch.cat(outs)
    (_, _, a), (_, _, b) = _operand(g, case, "lhs"), _operand(g, case, "rhs")
    a, b = a().double(), b().double()
    res = b @ a.t()
    if case["op"] == "train":
        dC = torch.randn(case["N"], case["M"], generator=g, device="cuda").double()
        return {"res": res, "dA": dC.t() @ b, "dB": dC @ a}
    return res.cpu() if case["op"] == "host" else res
