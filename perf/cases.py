"""Workloads of the correlator library, timed through its public Python calls.

Every case is one call that a user of the library makes again and again: a
correlation (uniform, raw packets, uneven and flagged channels, float
voltages in each precision mode), the adjoint of one, or a gain-calibration
gradient.  `listed()` holds the sizes of the library's own configurations and
benchmark legs and a few generic ones; `draw()` gives more of the same ranges.

A program of this kind keeps one handle for its lifetime and writes into
output buffers that it owns, so the handle is made once per process and the
outputs belong to the prepared state.  Calls are untuned, as the drop-in entry
points make them by default.
"""
import math

import torch

import ftd_b200
from ftd_b200 import Correlator, tri_size
from ftd_b200._lib import (COMPUTE_FP4, COMPUTE_FP8, COMPUTE_FP8_SPLIT, IN_FP16, IN_FP32, IN_INT4,
                           LAYOUT_TIME_ANT_CHAN_POL, OUT_FP16, OUT_FP32)

DEV = "cuda:0"
_handle = None


def corr():
    """The process's handle."""
    global _handle
    if _handle is None:
        _handle = Correlator(device=0)
    return _handle


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # a small array: 64 antennas x 2 polarisations, 32 channels, one short dump
        dict(name="qc_small", kind="qc", n=128, k=256, batch=32, out="f32"),
        # a mid-size array with sizes that are multiples of nothing, FP16 visibilities
        dict(name="qc_mid_odd_f16out", kind="qc", n=702, k=500, batch=24, out="f16"),
        # DSA-2000: 2048 antennas x 2 polarisations, 64 channels of 1024 samples
        dict(name="qc_large", kind="qc", n=4096, k=1024, batch=64, out="f32"),
        # few inputs, long integration: 128 antennas x 2 polarisations
        dict(name="qc_long", kind="qc", n=256, k=65536, batch=4, out="f32"),
        # voltages that were already FP16 (the FP16 drop-in call)
        dict(name="half_mid", kind="half", n=1024, k=1024, batch=16),
        # channels of uneven integration length with flagged inputs, one call
        dict(name="uneven", kind="uneven", rows=4096, chans=32, kmax=2048),
        # raw packets [t][ant][chan][pol] through the fused corner turn
        dict(name="packets", kind="packets", ant=2048, chan=16, pol=2, k=1024),
        # float voltages with RFI bursts, per-channel-scaled FP8
        dict(name="float_fp8", kind="float", n=4096, k=1024, batch=16, mode="fp8"),
        # the same voltages, hi + lo split FP8
        dict(name="float_split", kind="float", n=4096, k=1024, batch=16, mode="split"),
        # the same voltages, NVFP4
        dict(name="float_nvfp4", kind="float", n=4096, k=1024, batch=16, mode="nvfp4"),
        # backward of the correlator: dV = (G + G^H) V
        dict(name="adjoint", kind="adjoint", n=2048, k=512, batch=32),
        # gain calibration: loss and gradient over packed triangles
        dict(name="gain_gradient", kind="gain", n=2048, chans=32),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["qc", "qc", "qc", "long", "half", "uneven", "packets", "float", "float",
                       "float", "adjoint", "gain"])
    if kind == "qc":
        n, k = _log(rng, 100, 4096), _log(rng, 100, 2048)
        batch = _log(rng, 1, 64)
        return dict(kind="qc", n=n, k=k, batch=min(batch, _fit(n, k)), out=rng.choice(["f32", "f32", "f16"]))
    if kind == "long":
        n, k = _log(rng, 64, 512), _log(rng, 8192, 65536)
        return dict(kind="qc", n=n, k=k, batch=rng.randint(1, 8), out="f32")
    if kind == "half":
        n, k = _log(rng, 100, 2048), _log(rng, 100, 2048)
        return dict(kind="half", n=n, k=k, batch=min(_log(rng, 1, 32), _fit(n, k)))
    if kind == "uneven":
        return dict(kind="uneven", rows=_log(rng, 256, 4096), chans=rng.randint(2, 32),
                    kmax=64 * rng.randint(4, 32))
    if kind == "packets":
        return dict(kind="packets", ant=_log(rng, 100, 2048), chan=rng.randint(1, 16),
                    pol=rng.randint(1, 2), k=_log(rng, 100, 1024))
    if kind == "float":
        n, k = _log(rng, 200, 4096), _log(rng, 100, 1024)
        return dict(kind="float", n=n, k=k, batch=_log(rng, 1, 16),
                    mode=rng.choice(["fp8", "split", "nvfp4"]))
    if kind == "adjoint":
        return dict(kind="adjoint", n=8 * _log(rng, 16, 256), k=_log(rng, 64, 512),
                    batch=_log(rng, 1, 32))
    return dict(kind="gain", n=_log(rng, 100, 2048), chans=_log(rng, 1, 32))


def _fit(n, k):
    """Channels of n inputs x k samples that cost no more than the large case."""
    return max(1, int(64 * 4096 * 4096 * 1024 / (n * n * max(k, 1024))))


# ------------------------------------------------------------------ inputs
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _qc(shape, g):
    """QC bytes of complex Gaussian voltages (sigma 2.5 per part, rounded and
    clipped to [-7, 7]): high nibble Re, low nibble Im, sign-magnitude."""
    def nibble():
        v = torch.randn(shape, device=DEV, generator=g).mul_(2.5).round_().clamp_(-7, 7)
        return v.abs().to(torch.uint8) | ((v < 0).to(torch.uint8) << 3)
    out = nibble() << 4
    return out | nibble()


def _qc_complex(q):
    """QC bytes -> complex128."""
    def part(b):
        m = (b & 7).to(torch.float64)
        return torch.where((b & 8) != 0, -m, m)
    return torch.complex(part(q >> 4), part(q & 15))


def _float_voltages(b, n, k, g):
    """Complex Gaussian channels with an RMS log-uniform in [0.1, 10]; 1% of the
    samples carry 20-sigma bursts on 5% of the inputs."""
    rms = torch.exp(torch.empty(b, device=DEV).uniform_(math.log(0.1), math.log(10.0), generator=g))
    v = torch.randn(b, n, k, 2, device=DEV, generator=g) * (rms.view(b, 1, 1, 1) / math.sqrt(2.0))
    n_in, n_t = max(1, n // 20), max(1, k // 100)
    for c in range(b):
        ins = torch.randperm(n, device=DEV, generator=g)[:n_in]
        ts = torch.randperm(k, device=DEV, generator=g)[:n_t]
        ph = torch.rand(n_in, n_t, device=DEV, generator=g) * (2 * math.pi)
        v[c, ins[:, None], ts[None, :]] = 20.0 * rms[c] * torch.stack([torch.cos(ph), torch.sin(ph)], -1)
    return v


def _uneven(case, seed):
    """Per-channel (K, active inputs) of an uneven batch: K a multiple of 64 up
    to kmax, 37..100% of the inputs left after flagging."""
    cpu = torch.Generator().manual_seed(int(seed))
    rows = case["rows"]
    spec = []
    for _ in range(case["chans"]):
        k = 64 * int(torch.randint(2, case["kmax"] // 64 + 1, (1,), generator=cpu))
        n = int(torch.randint(max(1, rows * 3 // 8), rows + 1, (1,), generator=cpu))
        active = torch.sort(torch.randperm(rows, generator=cpu)[:n]).values.to(torch.int32)
        spec.append((k, n, active))
    return spec


def prepare(case, seed):
    kind, g = case["kind"], _gen(seed)
    s = dict(case)
    if kind == "qc":
        s["A"] = _qc((case["batch"], case["n"], case["k"]), g)
        dt = torch.float32 if case["out"] == "f32" else torch.float16
        s["C"] = torch.empty(case["batch"], tri_size(case["n"]), 2, device=DEV, dtype=dt)
    elif kind == "half":
        v = torch.randn(case["batch"], case["n"], case["k"], 2, device=DEV, generator=g)
        s["A"] = v.mul_(2.5).to(torch.float16)
        s["C"] = torch.empty(case["batch"], tri_size(case["n"]), 2, device=DEV, dtype=torch.float16)
    elif kind == "uneven":
        # the same channel geometry for every seed: a program's flags change, its channel plan
        # does not, and the work of a case is one number
        s["chans"] = [{"A": _qc((case["rows"], k), g), "n_inputs": n, "K": k, "active": active.to(DEV),
                       "C": torch.empty(tri_size(n), 2, device=DEV)}
                      for k, n, active in _uneven(case, 1)]
    elif kind == "packets":
        s["A"] = _qc((case["k"], case["ant"], case["chan"], case["pol"]), g)
        s["C"] = torch.empty(case["chan"] * case["pol"], tri_size(case["ant"]), 2, device=DEV)
    elif kind == "float":
        s["A"] = _float_voltages(case["batch"], case["n"], case["k"], g)
        s["C"] = torch.empty(case["batch"], tri_size(case["n"]), 2, device=DEV)
    elif kind == "adjoint":
        b, n, k = case["batch"], case["n"], case["k"]
        s["V"] = _qc((b, n, k), g)
        s["G"] = torch.randn(b, n, n, 2, device=DEV, generator=g)
        s["dV"] = torch.empty(b, n, k, 2, device=DEV)
    else:  # gain
        n, c = case["n"], case["chans"]
        p = tri_size(n)
        s["Rm"] = torch.randn(c, p, 2, device=DEV, generator=g).mul_(80.0)
        s["Ro"] = torch.randn(c, p, 2, device=DEV, generator=g).mul_(8.0).add_(s["Rm"])
        d = torch.arange(1, n + 1, device=DEV)
        d = d * (d + 1) // 2 - 1  # places of the autocorrelations
        s["Rm"][:, d] = torch.tensor([12800.0, 0.0], device=DEV)
        s["Ro"][:, d] = torch.tensor([12900.0, 0.0], device=DEV)
        s["W"] = torch.rand(c, p, device=DEV, generator=g)
        ph = torch.rand(n, device=DEV, generator=g) * (2 * math.pi)
        mag = 0.9 + 0.2 * torch.rand(n, device=DEV, generator=g)
        s["g"] = torch.stack([mag * torch.cos(ph), mag * torch.sin(ph)], -1).contiguous()
        s["grad"] = torch.empty(n, 2, device=DEV, dtype=torch.float64)
        s["loss"] = torch.empty(1, device=DEV, dtype=torch.float64)
    corr()
    return s


# ------------------------------------------------------------------ one pass
_MODES = {"fp8": COMPUTE_FP8, "split": COMPUTE_FP8_SPLIT, "nvfp4": COMPUTE_FP4}


def run(s):
    kind = s["kind"]
    if kind == "qc":
        call = ftd_b200.herk_batched_cutlass_qc if s["out"] == "f32" else ftd_b200.herk_batched_cutlass_qc_fp16
        call(s["A"], s["C"], s["n"], s["k"], s["batch"])
        return s["C"]
    if kind == "half":
        ftd_b200.herk_batched_cutlass_fp16(s["A"], s["C"], s["n"], s["k"], s["batch"])
        return s["C"]
    if kind == "uneven":
        corr().herk_batched_v(s["chans"], output=OUT_FP32)
        return [c["C"] for c in s["chans"]]
    if kind == "packets":
        corr().herk_ftd(s["A"], s["C"], s["ant"], s["chan"], s["pol"], s["k"],
                        layout=LAYOUT_TIME_ANT_CHAN_POL)
        return s["C"]
    if kind == "float":
        corr().herk(s["A"], s["C"], s["n"], s["k"], s["batch"], input=IN_FP32,
                    compute=_MODES[s["mode"]], output=OUT_FP32, tune=False)
        return s["C"]
    if kind == "adjoint":
        corr().herk_adjoint(s["G"], s["V"], s["dV"], s["n"], s["k"], s["batch"], input=IN_INT4)
        return s["dV"]
    corr().gain_gradient(s["Ro"], s["Rm"], s["W"], s["g"], s["n"], s["chans"], s["grad"], s["loss"])
    return {"grad": s["grad"], "loss": s["loss"]}


# ------------------------------------------------------------------ 64 bits
def _packed(v):
    """Packed lower triangle [n(n+1)/2][2] of v v^H for complex128 v [n][k]."""
    n = v.shape[0]
    r = v @ v.conj().T
    keep = torch.ones(n, n, dtype=torch.bool, device=v.device).tril_()
    return torch.view_as_real(r[keep])


def exact(case, seed):
    s = prepare(case, seed)
    kind = case["kind"]
    if kind == "qc":
        return torch.stack([_packed(_qc_complex(a)) for a in s["A"]])
    if kind in ("half", "float"):
        return torch.stack([_packed(torch.view_as_complex(a.double())) for a in s["A"]])
    if kind == "uneven":
        return [_packed(_qc_complex(c["A"][c["active"].long()])) for c in s["chans"]]
    if kind == "packets":
        v = _qc_complex(s["A"]).permute(2, 3, 1, 0).reshape(-1, case["ant"], case["k"])
        return torch.stack([_packed(a) for a in v])
    if kind == "adjoint":
        out = torch.empty(s["dV"].shape, dtype=torch.float64, device=DEV)
        for b in range(case["batch"]):
            gr = torch.view_as_complex(s["G"][b].double())
            out[b] = torch.view_as_real((gr + gr.conj().T) @ _qc_complex(s["V"][b]))
        return out
    n = case["n"]
    gains = torch.view_as_complex(s["g"].double())
    keep = torch.ones(n, n, dtype=torch.bool, device=DEV).tril_()
    grad = torch.zeros(n, dtype=torch.complex128, device=DEV)
    loss = torch.zeros(1, dtype=torch.float64, device=DEV)

    def full(p, dt):
        m = torch.zeros(n, n, dtype=dt, device=DEV)
        m[keep] = p
        low = m.tril(-1)
        return m + (low.conj().T if m.is_complex() else low.T)
    for c in range(case["chans"]):
        ro = full(torch.view_as_complex(s["Ro"][c].double()), torch.complex128)
        rm = full(torch.view_as_complex(s["Rm"][c].double()), torch.complex128)
        w = full(s["W"][c].double(), torch.float64)
        e = ro - gains[:, None] * rm * gains.conj()[None, :]
        loss += (w * e.abs().square()).sum()
        grad += -4.0 * (w * e * rm.conj()) @ gains
    return {"grad": torch.view_as_real(grad), "loss": loss}


# ------------------------------------------------------------------ cost
def work(case):
    kind = case["kind"]
    if kind in ("qc", "half", "float"):
        n, k, b = case["n"], case["k"], case["batch"]
        sample = {"qc": 1, "half": 4, "float": 8}[kind]
        out = 4 if kind == "half" or case.get("out") == "f16" else 8
        return {"bytes": b * (sample * n * k + out * tri_size(n)), "flops": 8 * b * tri_size(n) * k}
    if kind == "uneven":
        spec = _uneven(case, 1)
        return {"bytes": sum(n * k + 8 * tri_size(n) for k, n, _ in spec),
                "flops": sum(8 * tri_size(n) * k for k, n, _ in spec)}
    if kind == "packets":
        b, n, k = case["chan"] * case["pol"], case["ant"], case["k"]
        return {"bytes": b * (n * k + 8 * tri_size(n)), "flops": 8 * b * tri_size(n) * k}
    if kind == "adjoint":
        n, k, b = case["n"], case["k"], case["batch"]
        return {"bytes": b * (8 * n * n + n * k + 8 * n * k), "flops": 8 * b * n * n * k}
    n, c = case["n"], case["chans"]
    return {"bytes": c * tri_size(n) * 20 + 24 * n, "flops": 40 * c * tri_size(n)}


def tolerance(case):
    """Integer voltages give exact integers below 2^24, and FP16 roundings of
    them.  The others: FP32 sums of the same quantised products in another
    order (measured between the library's own kernels and split counts)."""
    kind = case["kind"]
    if kind in ("qc", "uneven", "packets"):
        return "exact"
    if kind == "half":  # FP16 results: another order of the sum moves some by one ulp
        return {"rel": 1e-4, "max": 4e-3}
    if kind == "float":  # K cut into four: 3.7e-6 in split mode, 6e-7 in plain FP8
        return {"rel": 1.5e-5, "max": 1e-3}
    if kind == "adjoint":
        return {"rel": 2e-5, "max": 1e-3}
    return {"rel": 1e-5, "max": 1e-4}
