"""What is timed when the speed of this codec is compared: the calls its users make, over the sizes they make them at.

Each case is one public entry point of ``trellis_b200`` at one size, number of bits per weight and codebook:

    encode     ``qtip.encode`` / ``qtip.viterbi_tb``: tiles in device memory -> codes (the plain quantiser's inner call)
    host       ``qtip.encode`` on pinned host tiles with pinned results (a checkpoint streamed through the GPU)
    rows       ``qtip.encode_rows``: one 16-row block of the LDLQ recursion, in place
    ldlq       ``ldlq.ldlq_b200``: the whole recursion of one matrix, packed codes out
    quantize   ``qtip.tcq_quantize_weight``: incoherence processing, encode, restore of one bf16 matrix
    ip         ``qtip.IPContext`` and its ``restore_tiles``: incoherence processing there and back
    decode     ``qtip.decode_packed``: code words -> weights
    matvec     ``qtip.decode_matvec``: products straight from code words (token generation from the packed model)
"""
from __future__ import annotations

import math
import os
import sys

import torch

_PKG = os.path.abspath("trellis-everywhere_b200")     # the folder users put on sys.path; the working folder is the repository's root
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from trellis_b200 import ldlq, qtip  # noqa: E402

CODEBOOKS = ("1mad", "3inst", "mcg")
DEV = "cuda"


def listed():
    return [
        # the smallest encodes: a handful of tiles, where the chain of 2 x 256 dependent steps is all there is
        {"name": "encode-8-k3", "kind": "encode", "n": 8, "K": 3, "cb": "3inst", "symbols": False},
        # a ragged batch through the drop-in call that also returns the symbols as int64
        {"name": "encode-1000-k2", "kind": "encode", "n": 1000, "K": 2, "cb": "mcg", "symbols": True},
        # one 4096 x 4096 matrix at 3 bits, the benchmark's workload
        {"name": "encode-65536-k3", "kind": "encode", "n": 65536, "K": 3, "cb": "3inst", "symbols": False},
        # the rate-distortion batch at 4 bits, from and to host memory
        {"name": "host-4096-k4", "kind": "host", "n": 4096, "K": 4, "cb": "1mad"},
        # one encoder call of LDLQ on a matrix with 4096 outputs: 256 tiles, the call such a quantisation makes hundreds of times
        {"name": "rows-4096-k3", "kind": "rows", "n_out": 4096, "K": 3, "cb": "mcg"},
        # a whole LDLQ recursion, 64 dependent encoder calls and their feedback products
        {"name": "ldlq-4096x1024-k3", "kind": "ldlq", "n_out": 4096, "k_in": 1024, "K": 3, "cb": "mcg"},
        # a key / value projection of the benchmark model, quantised as a checkpoint's bf16 matrix
        {"name": "quantize-1024x4096-k3", "kind": "quantize", "n_out": 1024, "k_in": 4096, "K": 3, "cb": "mcg"},
        # incoherence processing of a gate / up projection (larger than L2)
        {"name": "ip-12288x4096", "kind": "ip", "n_out": 12288, "k_in": 4096},
        # unpacking a few hundred tiles: launch latency
        {"name": "decode-300-k2", "kind": "decode", "n": 300, "K": 2, "cb": "3inst"},
        # unpacking a whole matrix of 67 M weights: memory bandwidth
        {"name": "decode-262144-k3", "kind": "decode", "n": 262144, "K": 3, "cb": "mcg"},
        # token generation, one sequence: a query / output projection
        {"name": "matvec-4096x4096-m1-k3", "kind": "matvec", "n_out": 4096, "k_in": 4096, "m": 1, "K": 3, "cb": "mcg"},
        # token generation, a few sequences together: the output head
        {"name": "matvec-151936x4096-m4-k4", "kind": "matvec", "n_out": 151936, "k_in": 4096, "m": 4, "K": 4, "cb": "3inst"},
    ]


def _log_int(rng, lo, hi):
    """An integer of [lo, hi], spread evenly over the logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    """One more case: the kind, bits per weight and codebook at random, sizes over the whole range of their kind."""
    kind = rng.choice(("encode", "encode", "encode", "host", "rows", "rows", "ldlq", "quantize", "ip", "decode", "decode", "matvec", "matvec"))
    c = {"kind": kind}
    if kind != "ip":
        c.update(K=rng.choice((2, 3, 4)), cb=rng.choice(CODEBOOKS))
    if kind == "encode":
        c.update(n=_log_int(rng, 1, 32768), symbols=rng.random() < 0.3)
    elif kind == "host":
        c.update(n=_log_int(rng, 16, 16384))
    elif kind == "rows":
        c.update(n_out=16 * _log_int(rng, 1, 768))
    elif kind == "ldlq":
        c.update(n_out=16 * _log_int(rng, 8, 256), k_in=16 * _log_int(rng, 8, 64))
    elif kind == "quantize":
        c.update(n_out=16 * _log_int(rng, 4, 256), k_in=16 * _log_int(rng, 4, 128))
    elif kind == "ip":
        n_out = 16 * _log_int(rng, 4, 768)
        c.update(n_out=n_out, k_in=16 * _log_int(rng, 4, min(768, (12288 * 4096) // (16 * n_out))))
    elif kind == "decode":
        c.update(n=_log_int(rng, 1, 400000))
    else:
        n_out = 16 * _log_int(rng, 4, 9496)
        c.update(n_out=n_out, k_in=16 * _log_int(rng, 4, min(768, (151936 * 4096) // (16 * n_out))), m=rng.choice((1, 1, 2, 3, 4, 5, 8)))
    return c


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _cb_rms(cb):
    return qtip.codebook_lut(cb, DEV).square().mean().sqrt().item()


def _words(n, K, g):
    """Every bit pattern is a valid tail-biting code stream, and codes of real weights are close to uniform."""
    return torch.randint(-2 ** 31, 2 ** 31, (n, 8 * K), dtype=torch.int64, generator=g, device=DEV).to(torch.int32)


def _weights(n_out, k_in, g):
    """N(0, 0.02^2) with 1 % outliers x 20, as the benchmark matrix."""
    w = torch.randn(n_out, k_in, generator=g, device=DEV) * 0.02
    return torch.where(torch.rand(n_out, k_in, generator=g, device=DEV) < 0.01, w * 20, w)


def prepare(case, seed):
    g, kind, s = _gen(seed), case["kind"], {"case": case, "seed": seed}
    if kind in ("encode", "host"):
        # incoherence-processed weights are Gaussian with the codebook's RMS
        w = torch.randn(case["n"], qtip.T_SEQ, generator=g, device=DEV) * _cb_rms(case["cb"])
        if kind == "encode":
            s["w"] = w
        else:
            n, pin = case["n"], {"pin_memory": True}
            s["w"] = torch.empty(n, qtip.T_SEQ, **pin).copy_(w)
            s["out"] = qtip.Encoded(torch.empty(n, 8 * case["K"], dtype=torch.int32, **pin), torch.empty(n, qtip.T_SEQ, **pin),
                                    torch.empty(n, **pin), None)
    elif kind == "rows":
        n = case["n_out"]
        s["src"] = torch.randn(16, n, generator=g, device=DEV) * _cb_rms(case["cb"])
        s["comp"] = torch.randn(16, n, generator=g, device=DEV) * 0.1
        s["wq"], s["err"] = torch.empty_like(s["src"]), torch.empty_like(s["src"])
        s["packed"] = torch.empty(n // 16, 8 * case["K"], dtype=torch.int32, device=DEV)
        s["sse"] = torch.empty(n // 16, device=DEV)
    elif kind == "ldlq":
        n, k = case["n_out"], case["k_in"]
        s["wt"] = torch.randn(k, n, generator=g, device=DEV) * _cb_rms(case["cb"])
        # the proxy Hessian of Gaussian activations with per-channel scales log-uniform in [0.1, 10], factored once per matrix
        scales = torch.exp(torch.empty(k, device=DEV).uniform_(math.log(0.1), math.log(10.0), generator=g))
        x = torch.randn(2 * k, k, generator=g, device=DEV) * scales
        s["L"] = ldlq.block_ldl(ldlq.regularize_H(x.t() @ x / (2 * k)))
        s["packed"] = torch.empty(n // 16, k // 16, 8 * case["K"], dtype=torch.int32, device=DEV)
    elif kind == "quantize":
        s["w"] = _weights(case["n_out"], case["k_in"], g).to(torch.bfloat16)
    elif kind == "ip":
        s["w"], s["cb_rms"] = _weights(case["n_out"], case["k_in"], g), _cb_rms("mcg")
    elif kind == "decode":
        s["packed"] = _words(case["n"], case["K"], g)
    else:
        s["packed"] = _words(case["n_out"] // 16 * (case["k_in"] // 16), case["K"], g)
        s["x"] = torch.randn(case["m"], case["k_in"], generator=g, device=DEV)
    return s


def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind == "encode":
        if c["symbols"]:
            return qtip.viterbi_tb(s["w"], c["K"], c["cb"])
        return tuple(qtip.encode(s["w"], c["K"], c["cb"]))
    if kind == "host":
        return tuple(qtip.encode(s["w"], c["K"], c["cb"], out=s["out"]))
    if kind == "rows":
        qtip.encode_rows(s["src"], s["comp"], c["K"], c["cb"], s["wq"], s["err"], s["packed"], s["sse"])
        return s["wq"], s["err"], s["packed"], s["sse"]
    if kind == "ldlq":
        return ldlq.ldlq_b200(s["wt"], s["L"], c["K"], c["cb"], packed=s["packed"]), s["packed"]
    if kind == "quantize":
        return qtip.tcq_quantize_weight(s["w"], c["K"], c["cb"], seed=s["seed"])
    if kind == "ip":
        ip = qtip.IPContext(s["w"], s["cb_rms"], seed=s["seed"])
        return ip.tiles, ip.out_s, ip.in_s, ip.restore_tiles(ip.tiles)
    if kind == "decode":
        return qtip.decode_packed(s["packed"], c["K"], c["cb"])
    return qtip.decode_matvec(s["packed"], c["n_out"], c["k_in"], c["K"], c["cb"], s["x"])


# Two passes of 65 536 state evaluations per weight, each a subtraction, a multiplication, an addition and a comparison.
_ENCODE_OPS = 2 * 65536 * 4


def work(case):
    kind, K = case["kind"], case.get("K", 0)
    if kind in ("encode", "host"):
        weights = case["n"] * qtip.T_SEQ
        out = weights * (8 + 4) if case.get("symbols") else weights * (4 + K / 8) + 4 * case["n"]
        return {"bytes": weights * 4 + out, "flops": weights * _ENCODE_OPS}
    if kind == "rows":
        weights = 16 * case["n_out"]
        return {"bytes": weights * (4 * 4 + K / 8) + case["n_out"] / 4, "flops": weights * _ENCODE_OPS}
    if kind == "decode":
        weights = case["n"] * qtip.T_SEQ
        return {"bytes": weights * (4 + K / 8), "flops": weights * 8}       # unpack, scramble and convert
    weights = case["n_out"] * case["k_in"]
    if kind == "ldlq":
        return {"bytes": weights * (4 + 4 + K / 8) + 4 * case["k_in"] ** 2, "flops": weights * (_ENCODE_OPS + case["k_in"])}
    if kind == "quantize":
        return {"bytes": weights * (2 + 2), "flops": weights * (_ENCODE_OPS + 2 * 2 * 7)}
    if kind == "ip":
        # there and back: one read and one write each; seven butterfly stages on each axis, each way
        return {"bytes": weights * 4 * 4, "flops": weights * 2 * 2 * 7}
    return {"bytes": weights * K / 8 + 4 * case["m"] * (case["n_out"] + case["k_in"]), "flops": weights * (8 + 2 * case["m"])}


def tolerance(case):
    """Codes, reconstructions of given codes and path costs are bit-exact by contract.  The others, about four times what
    the same steps in fp64 differ by:

    ip        fp32 transforms and sums (measured: 1.9e-7, largest 3.1e-6)
    quantize  one or two tiles in 16 384 sit on a near-tie that the last ulp of their incoherence-processed weights
              decides; such a tile moves the result by 0.23 / sqrt(tiles) of its norm (measured: 1.8e-3 at 16 384 tiles,
              largest 0.15 where the inverse transform spreads it over a 128 x 128 block)
    matvec    fp32 dot products (measured: 4.8e-7, largest 1.5e-6)
    """
    if case["kind"] == "ip":
        return {"rel": 8e-7, "max": 1.3e-5}
    if case["kind"] == "quantize":
        return {"rel": min(0.03, 0.9 / math.sqrt(case["n_out"] * case["k_in"] / 256)), "max": 0.6}
    if case["kind"] == "matvec":
        return {"rel": 2e-6, "max": 6e-6}
    return "exact"
