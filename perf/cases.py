"""Performance cases of focss_gb300: the calls a user of the framework makes,
at the sizes of its own configurations and around them.

Links: 32 GBaud 16QAM over spans of standard single-mode fibre (0.2 dB/km,
17 ps/nm/km, 1.3 /W/km) with EDFAs.  Six families:

  fwd     forward propagation (single channel, WDM, dual polarization)
  dbp     digital back-propagation of a sweep of lengths and steps per span
  tx, rx  transmitter and receiver chains, decide: decisions and scores
  ppe     perturbation (triplet) equalizers, and the fit of their coefficients
  ldbp    learned back-propagation, receiving and training
  cnn     training of the correction network behind it

`listed()` are the cases that are always measured, `draw(rng)` gives others of
the same ranges.  Inputs are synthetic and a function of the seed alone;
`exact` restates each case in 64 bits with torch.
"""
import math

import numpy as np
import torch

import focss_gb300 as fg
from focss_gb300 import dsp, sino
from focss_gb300.cnn import CorrectionCNN
from focss_gb300.ldbp import LearnedDBP

DEV = "cuda"
C128 = torch.complex128
LIGHT = 299792458.0
WAVELENGTH = 1.55e-6
F0 = LIGHT / WAVELENGTH
PLANCK = 6.62607004081818181818181e-34
BAUD = 32e9
ALPHA = 0.2e-3 * math.log(10) / 10
BETA2 = -WAVELENGTH * WAVELENGTH * 17e-6 / (2 * math.pi * LIGHT)
GAMMA = 1.3e-3
SPACING = 50e9
ROLL_OFF = 0.1
CNN_LAYERS = ((16, 64), (64, 64), (64, 64), (64, 16))  # (inputs, outputs) of the 9-tap convolutions
CNN_TRIPLETS = ((0, 0), (0, 1), (0, 2), (0, 3), (1, 1), (1, -1), (1, 2))


def listed():
    return [
        # One single-channel field of 2^14 symbols at 8 samples per symbol over
        # spans of fixed 1 km steps: the latency of one simulation.
        dict(name="fwd_single", kind="fwd", samples=2 ** 17, modes=1, batch=1, channels=1, osf=8, grid="uniform",
             steps=80, spans=4, span_m=80e3, power_lo=2.0, power_hi=2.0, nf_db=0.0, kappa=1.0),
        # The precision study: 5 WDM channels of 2^15 symbols, a launch-power
        # sweep of 28 realizations, phase-bounded steps and ASE.  The largest case.
        dict(name="fwd_wdm", kind="fwd", samples=2 ** 19, modes=1, batch=28, channels=5, osf=16, grid="adaptive",
             phase=0.005, spans=1, span_m=80e3, power_lo=-2.0, power_hi=4.0, nf_db=5.0, kappa=1.0),
        # One dual-polarization WDM realization (Manakov), as a dataset is generated.
        dict(name="fwd_dualpol", kind="fwd", samples=2 ** 19, modes=2, batch=1, channels=3, osf=16, grid="adaptive",
             phase=0.001, spans=1, span_m=100e3, power_lo=2.0, power_hi=2.0, nf_db=4.5, kappa=8.0 / 9.0),
        # Back-propagation of the batched sweep: five lengths at 1..16 steps
        # per span, 25 fields of uneven length in one call.
        dict(name="dbp_sweep", kind="dbp", log2_lo=13, log2_hi=17, batch=5, steps_max=16, spans=15),
        # A 5-channel WDM transmitter from symbol codes in host memory.
        dict(name="tx_wdm", kind="tx", symbols=2 ** 15, channels=5, osf=16, modes=1),
        # The centre channel's receiver for a batch of received WDM fields.
        dict(name="rx_wdm", kind="rx", symbols=2 ** 15, batch=12, osf=16, channels=5, spans=20),
        # Decisions and scores of one short received sequence: the smallest calls.
        dict(name="decide_small", kind="decide", symbols=4000, modes=1, batch=1),
        # Triplet equalizer of radius 75 on 2^20 symbols, coefficients pruned.
        dict(name="ppe_r75", kind="ppe", symbols=2 ** 20, modes=1, radius=75, keep=0.999),
        # Dual-polarization WDM equalizer (self- and cross-phase terms) on one dataset.
        dict(name="ppe_wdm", kind="ppe_wdm", symbols=2 ** 15, batch=1, c=30, d=3),
        # Learned back-propagation, 4 steps per span, as a receiver.
        dict(name="ldbp_rx", kind="ldbp", symbols=2 ** 15, batch=16, spans=20, steps=4, taps=63, mf_taps=255,
             train=False),
        # One training step's loss and gradients of that model.
        dict(name="ldbp_train", kind="ldbp", symbols=2 ** 15, batch=16, spans=20, steps=4, taps=63, mf_taps=255,
             train=True),
        # The same of the correction network, on three quarters of the batch.
        dict(name="cnn_train", kind="cnn", symbols=2 ** 15, batch=12, train=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["fwd", "fwd", "dbp", "tx", "rx", "decide", "ppe", "ppe_wdm", "ppe_fit", "ldbp", "ldbp", "cnn"])
    if kind == "fwd":
        lg, modes = rng.randint(12, 19), rng.choice([1, 1, 2])
        grid = rng.choice(["uniform", "adaptive", "logarithmic"])
        most = min(64 if grid == "logarithmic" else 256, 2 ** (22 - lg) * 3 // modes)
        c = dict(kind=kind, samples=2 ** lg, modes=modes, batch=_log(rng, 1, most),
                 channels=1 if lg < 15 else rng.choice([1, 3, 5]), osf=16, grid=grid, spans=1, span_m=80e3,
                 power_lo=-2.0, power_hi=rng.choice([0.0, 2.0, 4.0]), nf_db=rng.choice([0.0, 5.0]),
                 kappa=8.0 / 9.0 if modes == 2 else 1.0)
        if grid == "uniform":
            c["steps"] = rng.randint(20, 160)
        else:
            c["phase"] = rng.choice([0.005, 0.01])
        return c
    if kind == "dbp":
        lo = rng.randint(12, 15)
        return dict(kind=kind, log2_lo=lo, log2_hi=rng.randint(lo, 17), batch=_log(rng, 1, 7),
                    steps_max=rng.choice([1, 4, 8, 16]), spans=rng.randint(5, 15))
    if kind == "tx":
        return dict(kind=kind, symbols=2 ** rng.randint(11, 15), channels=rng.choice([1, 3, 5]), osf=rng.choice([8, 16]),
                    modes=rng.choice([1, 2]))
    if kind == "rx":
        return dict(kind=kind, symbols=2 ** rng.randint(11, 15), batch=_log(rng, 1, 12), osf=16,
                    channels=rng.choice([3, 5]), spans=rng.randint(5, 20))
    if kind == "decide":
        return dict(kind=kind, symbols=_log(rng, 1000, 300000), modes=rng.choice([1, 2]), batch=_log(rng, 1, 16))
    if kind == "ppe":
        return dict(kind=kind, symbols=_log(rng, 30000, 1000000), modes=rng.choice([1, 1, 2]), radius=rng.randint(8, 75),
                    keep=rng.choice([1.0, 0.999, 0.5]))
    if kind == "ppe_wdm":
        return dict(kind=kind, symbols=_log(rng, 5000, 200000), batch=rng.randint(1, 2), c=rng.randint(8, 36),
                    d=rng.randint(0, 6))
    if kind == "ppe_fit":
        return dict(kind=kind, symbols=_log(rng, 10000, 40000), c=rng.randint(8, 30), d=rng.randint(0, 3))
    if kind == "ldbp":
        return dict(kind=kind, symbols=_log(rng, 3000, 33000), batch=_log(rng, 1, 16), spans=rng.choice([10, 20]),
                    steps=rng.randint(2, 4), taps=2 * rng.randint(7, 31) + 1, mf_taps=2 * rng.randint(31, 127) + 1,
                    train=rng.random() < 0.6)
    return dict(kind=kind, symbols=_log(rng, 3000, 33000), batch=_log(rng, 1, 12), train=rng.random() < 0.6)


# ---------------------------------------------------------------- fields and tensors
class _Device:
    """A field's device memory as an array that torch reads; keeps the field."""

    def __init__(self, field):
        self.field = field
        self.__cuda_array_interface__ = {"shape": (*field.shape, 2), "typestr": "<f4", "strides": None, "version": 3,
                                         "data": (int(field.device_ptr()), False)}


def _tensor(field):
    return torch.view_as_complex(torch.as_tensor(_Device(field), device=DEV))


def _field(values, dt):
    """A new field holding `values` (batch x modes x samples on the GPU)."""
    f = fg.Field(fg.Domain(values.shape[1], values.shape[2], dt, F0), batch=values.shape[0])
    f.ctx.sync()
    _tensor(f).copy_(values)
    torch.cuda.synchronize()
    return f


# ---------------------------------------------------------------- inputs
def _rng(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _randn(g, *shape):
    return torch.complex(torch.randn(shape, generator=g, device=DEV, dtype=torch.float64),
                         torch.randn(shape, generator=g, device=DEV, dtype=torch.float64)) * math.sqrt(0.5)


def _qam(g, *shape):
    """16QAM symbols of unit average power."""
    levels = torch.randint(0, 4, (2, *shape), generator=g, device=DEV).double() * 2 - 3
    return torch.complex(levels[0], levels[1]) / math.sqrt(10.0)


def _shaped(sym, osf, spacing):
    """Root-raised-cosine WDM waveforms (batch x modes x samples) of unit power
    per channel from sym[batch, channel, mode, symbols]."""
    _, nch, _, ns = sym.shape
    n = ns * osf
    f = torch.fft.fftfreq(n, 1.0 / (osf * BAUD), device=DEV, dtype=torch.float64).abs()
    edge = ((f / BAUD - (1 - ROLL_OFF) / 2) / ROLL_OFF).clamp(0, 1)
    h = torch.cos(0.5 * math.pi * edge)
    out = torch.zeros(sym.shape[0], sym.shape[2], n, dtype=C128, device=DEV)
    for c in range(nch):
        s = torch.fft.fft(sym[:, c]).repeat(1, 1, osf) * h
        out += torch.roll(s, round((c - nch // 2) * spacing * ns / BAUD), dims=-1)
    return torch.fft.ifft(out) * osf


def _omega2(n, dt):
    w = 2 * math.pi * torch.fft.fftfreq(n, dt, device=DEV, dtype=torch.float64)
    return w * w


def _dispersed(x, dt, length):
    return torch.fft.ifft(torch.fft.fft(x) * torch.polar(torch.ones((), dtype=torch.float64, device=DEV),
                                                         0.5 * BETA2 * length * _omega2(x.shape[-1], dt)))


def _watts(dbm):
    return 1e-3 * 10 ** (dbm / 10)


def _fwd_input(c, seed):
    g = _rng(seed)
    sym = _qam(g, c["batch"], c["channels"], c["modes"], c["samples"] // c["osf"])
    p = torch.linspace(c["power_lo"], c["power_hi"], c["batch"], device=DEV, dtype=torch.float64)
    return (_shaped(sym, c["osf"], SPACING) * torch.sqrt(_watts(p) / c["modes"]).view(-1, 1, 1)).to(torch.complex64)


def _dbp_inputs(c, seed):
    """Received fields at 2 samples per symbol, one per length."""
    g = _rng(seed)
    out = []
    for lg in range(c["log2_lo"], c["log2_hi"] + 1):
        x = _shaped(_qam(g, c["batch"], 1, 1, 2 ** (lg - 1)), 2, SPACING) * math.sqrt(_watts(1.0))
        x = _dispersed(x, 1 / (2 * BAUD), 80e3 * c["spans"]) + _randn(g, *x.shape) * math.sqrt(_watts(-18.0))
        out.append(x.to(torch.complex64))
    return out


def _dbp_steps(c):
    return [k for k in (1, 2, 4, 8, 16) if k <= c["steps_max"]]


def _rx_input(c, seed):
    g = _rng(seed)
    sym = _qam(g, c["batch"], c["channels"], 1, c["symbols"]) * math.sqrt(_watts(0.0))
    x = _dispersed(_shaped(sym, c["osf"], SPACING), 1 / (BAUD * c["osf"]), 80e3 * c["spans"])
    x = x * np.exp(0.7j) + _randn(g, *x.shape) * math.sqrt(_watts(-8.0))
    return x.to(torch.complex64), sym[:, c["channels"] // 2].to(torch.complex64)


def _noisy_symbols(c, seed, batch, modes, noise):
    g = _rng(seed)
    tx = _qam(g, batch, modes, c["symbols"])
    rx = tx * (1 + 0.02j * (tx.abs() ** 2 - 1)) + noise * _randn(g, *tx.shape)
    return tx.to(torch.complex64), rx.to(torch.complex64)


def _table(seed, radius, scale):
    """Coefficients that fall off from the centre as perturbation terms do, the
    products |m n| weighting them, (2R+1)^2."""
    rng = np.random.default_rng(seed)
    m, n = np.meshgrid(np.arange(-radius, radius + 1), np.arange(-radius, radius + 1), indexing="ij")
    mag = scale / (1.0 + np.abs(m * n) + 0.2 * (np.abs(m) + np.abs(n)))
    return mag * np.exp(2j * np.pi * rng.random(m.shape))


def _ppe_terms(c, seed):
    """Term list of the diamond |m| + |n| <= radius, the weakest dropped."""
    r = c["radius"]
    m, n = (v.ravel().astype(np.int32) for v in np.meshgrid(np.arange(-r, r + 1), np.arange(-r, r + 1), indexing="ij"))
    inside = np.abs(m) + np.abs(n) <= r
    m, n, k = m[inside], n[inside], _table(seed, r, 4e-3).ravel()[inside]
    keep = np.argsort(-np.abs(k), kind="stable")[:max(1, int(c["keep"] * k.size))]
    keep.sort()
    return m[keep], n[keep], k[keep]


def _rrc_pulse(n_symbols, osf, roll_off):
    """Time-domain root-raised-cosine pulse with sum h^2 = length."""
    t = np.arange(n_symbols * osf) / osf - n_symbols / 2.0
    h = np.empty_like(t)
    q = np.abs(t) == 1 / roll_off / 4
    z = t == 0
    o = ~(z | q)
    h[z] = 1 - roll_off + 4 * roll_off / np.pi
    h[q] = roll_off / np.sqrt(2) * ((1 + 2 / np.pi) * np.sin(np.pi / roll_off / 4) +
                                    (1 - 2 / np.pi) * np.cos(np.pi / roll_off / 4))
    u = t[o]
    h[o] = (np.cos(np.pi * u * (1 + roll_off)) * 4 * roll_off * u + np.sin(np.pi * u * (1 - roll_off))) / (
        (1 - 16 * roll_off ** 2 * u ** 2) * np.pi * u)
    return h * (h.size / np.sum(h * h))


def _ldbp_params(c):
    """Split-step back-propagation as the learned model's initial parameters."""
    n, dt, step = 2 * c["symbols"], 1 / (2 * BAUD), 80e3 / c["steps"]
    w2 = (2 * np.pi * np.fft.fftfreq(n, dt)) ** 2

    def response(length):
        return np.exp(0.5 * ALPHA * length) * np.exp(-0.5j * BETA2 * length * w2)

    def taps(resp, count):
        half = (count - 1) // 2
        return (np.fft.fft(resp) / n)[np.arange(-half, half + 1) % n]

    layers = c["spans"] * c["steps"]
    h = np.tile(taps(response(step), c["taps"]), (layers, 1))
    h[0] = taps(response(step / 2), c["taps"])
    edge = np.clip((np.abs(np.fft.fftfreq(n, dt)) / BAUD - (1 - ROLL_OFF) / 2) / ROLL_OFF, 0, 1)
    hmf = taps(np.cos(0.5 * np.pi * edge) * response(step / 2), c["mf_taps"])
    return (h.astype(np.complex64), np.full(layers, -GAMMA * step, np.float32), hmf.astype(np.complex64))


def _ldbp_input(c, seed):
    g = _rng(seed)
    sym = _qam(g, c["batch"], 1, 1, c["symbols"]) * math.sqrt(_watts(1.0))
    x = _dispersed(_shaped(sym, 2, SPACING), 1 / (2 * BAUD), 80e3 * c["spans"])
    x = x + _randn(g, *x.shape) * math.sqrt(_watts(-14.0))
    return x.to(torch.complex64), sym[:, 0].to(torch.complex64)


def _cnn_params(seed):
    rng = np.random.default_rng(seed)
    out = []
    for i, (cin, cout) in enumerate(CNN_LAYERS):
        w = rng.standard_normal((cout, 9, cin)) * math.sqrt(2.0 / (9 * cin))
        if i == 3:
            w[2:] = 0
            w *= 0.05
        out += [w.ravel(), 0.01 * rng.standard_normal(cout) * (i < 3)]
    return np.concatenate(out).astype(np.float32)


# ---------------------------------------------------------------- prepare and run
def _fiber(c):
    return fg.Fiber(ALPHA, BETA2, GAMMA, c.get("span_m", 80e3), WAVELENGTH, c.get("kappa", 1.0))


def _gain(c):
    return math.exp(ALPHA * c.get("span_m", 80e3))


def _ssfm(c):
    s = fg.SSFM(_fiber(c))
    s.set_grid({"uniform": fg.SSFM.UNIFORM, "logarithmic": fg.SSFM.LOGARITHMIC, "adaptive": fg.SSFM.ADAPTIVE}[c["grid"]])
    if c["grid"] == "uniform":
        s.set_total_steps(c["steps"])
    else:
        s.set_maximum_phase_shift(c["phase"])
        s.set_maximum_step_size(1000.0)
    return s


def prepare(case, seed):
    c, st = case, {"case": case}
    kind = c["kind"]
    if kind == "fwd":
        st["src"] = _field(_fwd_input(c, seed), 1 / (BAUD * c["osf"]))
        st["f"] = st["src"].copy()
        st["out"] = _tensor(st["f"])
        st["ssfm"] = _ssfm(c)
        st["amp"] = fg.Amplifier(_gain(c), 10 ** (c["nf_db"] / 10) if c["nf_db"] else 0.0, seed=seed)
    elif kind == "dbp":
        st["src"] = [_field(x, 1 / (2 * BAUD)) for x in _dbp_inputs(c, seed)]
        ks = _dbp_steps(c)
        st["f"] = [f.copy() for _ in ks for f in st["src"]]
        st["ssfm"] = [fg.SSFM(_fiber(c), k) for k in ks for _ in st["src"]]
        st["amp"] = fg.Amplifier(_gain(c))
        st["out"] = [_tensor(f) for f in st["f"]]
    elif kind == "tx":
        rng = np.random.default_rng(seed)
        st["codes"] = rng.integers(0, 16, (c["channels"], c["modes"], c["symbols"])).astype(np.int32)
    elif kind == "rx":
        x, t = _rx_input(c, seed)
        st["f"], st["tx"] = _field(x, 1 / (BAUD * c["osf"])), _field(t, 1 / BAUD)
        st["pse"] = dsp.PhaseShiftEqualizer(720)
    elif kind == "decide":
        t, r = _noisy_symbols(c, seed, c["batch"], c["modes"], 0.2)
        st["tx"], st["rx"] = _field(t, 1 / BAUD), _field(r, 1 / BAUD)
    elif kind == "ppe":
        t, _ = _noisy_symbols(c, seed, 1, c["modes"], 0.1)
        st["tx"] = _field(t * math.sqrt(0.5), 1 / BAUD)
        st["terms"] = _ppe_terms(c, seed)
    elif kind == "ppe_wdm":
        t, r = _noisy_symbols(c, seed, c["batch"], 6, 0.1)
        st["tx"], st["rx"] = _field(t, 1 / BAUD), _field(r, 1 / BAUD)
        st["ppe"] = fg.WdmPPE(c["c"], c["d"]).set_tables(_table(seed, c["c"], 4e-3), _table(seed + 1, c["d"], 4e-3),
                                                       0.98 + 0.05j)
    elif kind == "ppe_fit":
        t, r = _noisy_symbols(c, seed, 1, 6, 0.1)
        st["tx"], st["rx"] = _field(t, 1 / BAUD), _field(r, 1 / BAUD)
        st["ppe"] = fg.WdmPPE(c["c"], c["d"])
    elif kind == "ldbp":
        x, t = _ldbp_input(c, seed)
        st["f"], st["tx"] = _field(x, 1 / (2 * BAUD)), _field(t, 1 / BAUD)
        m = LearnedDBP(c["spans"], c["steps"], c["taps"], c["mf_taps"], 2 * c["symbols"], c["batch"],
                       _gain(c) ** -0.5)
        m.set_params(*_ldbp_params(c))
        st["model"] = m
    else:
        t, r = _noisy_symbols(c, seed, c["batch"], 1, 0.1)
        st["tx"], st["rx"] = _field(t, 1 / BAUD), _field(r, 1 / BAUD)
        m = CorrectionCNN(c["symbols"], c["batch"], 1.0, triplets=CNN_TRIPLETS)
        m.set_params(_cnn_params(seed))
        st["model"] = m
    return st


def run(state):
    st, c = state, state["case"]
    kind = c["kind"]
    if kind == "fwd":
        st["f"].assign(st["src"])
        if c["grid"] == "adaptive":
            fg.span_loop([st["f"]], _fiber(c), st["ssfm"], c["spans"], after=fg.Amplifier.AMPLIFY, amplifier=st["amp"])
        else:
            fg.forward_propagation(st["f"], _fiber(c), st["ssfm"], st["amp"], c["spans"])
        return st["out"]
    if kind == "dbp":
        n = len(st["src"])
        for i, f in enumerate(st["f"]):
            f.assign(st["src"][i % n])
        fg.span_loop(st["f"], _fiber(c), st["ssfm"], c["spans"], direction=fg.SSFM.BACKWARD, amplifier=st["amp"],
                     before=fg.Amplifier.DROP_POWER)
        return st["out"]
    if kind == "tx":
        sym = dsp.qam16_map(st["codes"], fg.Domain(c["modes"], c["symbols"], 1 / BAUD, F0), batch=c["channels"])
        sym *= math.sqrt(_watts(0.0) / c["modes"])
        return _tensor(dsp.wdm_mux(dsp.rrc_shaping(sym, c["osf"], ROLL_OFF), SPACING))
    if kind == "rx":
        f = dsp.decimate(dsp.wdm_select(st["f"], 0, SPACING), c["osf"] // 2)
        fg.cd_compensation(f, _fiber(c), c["spans"])
        return _tensor(st["pse"].train_equalize(st["tx"], dsp.rrc_sampling(f, 2, ROLL_OFF)))
    if kind == "decide":
        return {"hard": _tensor(dsp.hard_decision_16qam(st["rx"])), "codes": dsp.hd_sequence_16qam(st["rx"]),
                "ber": dsp.bit_error_rate_16qam(st["tx"], st["rx"]), "q2": dsp.q2_factor(st["tx"], st["rx"])}
    if kind == "ppe":
        return _tensor(sino.triplet_apply(st["tx"], c["radius"], *st["terms"]))
    if kind == "ppe_wdm":
        return _tensor(st["ppe"].equalize(st["tx"], st["rx"]))
    if kind == "ppe_fit":
        p = st["ppe"].train(st["tx"], st["rx"])
        return {"C": p.C, "D": p.D, "linear": np.complex128(p.linear_weight)}
    if kind == "ldbp":
        if not c["train"]:
            return _tensor(st["model"].forward(st["f"]))
        loss = st["model"].loss_grad(st["f"], st["tx"])
        h, xi, hmf = st["model"].get_params()[1]
        return {"loss": loss, "h": h.astype(np.complex64), "xi": xi.astype(np.float32), "hmf": hmf.astype(np.complex64)}
    if not c["train"]:
        return _tensor(st["model"].forward(st["rx"]))
    loss = st["model"].loss_grad(st["rx"], st["tx"])
    return {"loss": loss, "grads": st["model"].get_params()[1]}


# ---------------------------------------------------------------- work
def _fwd_steps(c):
    """Split steps per span: counted for a uniform grid, estimated for the
    others from the launch power (peak about 10 times the mean) and the loss."""
    if c["grid"] == "uniform":
        return c["steps"]
    p = _watts(0.5 * (c["power_lo"] + c["power_hi"])) * c["channels"] * 10
    z = (np.arange(1000) + 0.5) / 1000 * c["span_m"]
    rate = GAMMA * c["kappa"] * p * np.exp(-ALPHA * z) / c["phase"]
    return float(np.sum(np.maximum(rate, 1e-3)) * c["span_m"] / 1000)


def work(case):
    c = case
    kind = c["kind"]
    if kind == "fwd":
        n = c["batch"] * c["modes"] * c["samples"]
        return {"bytes": 16.0 * n, "flops": n * c["spans"] * _fwd_steps(c) * (10 * math.log2(c["samples"]) + 20)}
    if kind == "dbp":
        ks = _dbp_steps(c)
        ns = [2.0 ** lg * c["batch"] for lg in range(c["log2_lo"], c["log2_hi"] + 1)]
        return {"bytes": 16.0 * sum(ns) * len(ks),
                "flops": sum(n * (10 * math.log2(n / c["batch"]) + 20) for n in ns) * sum(ks) * c["spans"]}
    if kind == "tx":
        n = c["symbols"] * c["osf"] * c["modes"]
        return {"bytes": 4.0 * c["symbols"] * c["channels"] * c["modes"] + 8.0 * n,
                "flops": n * c["channels"] * (10 * math.log2(c["symbols"] * c["osf"]) + 20)}
    if kind == "rx":
        n = c["symbols"] * c["osf"] * c["batch"]
        return {"bytes": 8.0 * n + 16.0 * c["symbols"] * c["batch"],
                "flops": n * 10 * math.log2(c["symbols"] * c["osf"])}
    if kind == "decide":
        n = c["symbols"] * c["modes"] * c["batch"]
        return {"bytes": 28.0 * n, "flops": 60.0 * n}
    if kind == "ppe":
        r = c["radius"]
        terms = c["keep"] * (2 * r * (r + 1) + 1)
        n = c["symbols"] * c["modes"]
        return {"bytes": 16.0 * n, "flops": 8.0 * terms * c["symbols"] + 16.0 * n * (2 * r + 1)}
    if kind == "ppe_wdm":
        n = c["symbols"] * c["batch"]
        spm, xpm = 2 * c["c"] * (c["c"] + 1) + 1, 2 * c["d"] * (c["d"] + 1) + 1
        return {"bytes": 8.0 * n * 10, "flops": n * (8.0 * spm + 14 * 8.0 * xpm)}
    if kind == "ppe_fit":
        nf = c["c"] * (c["c"] + 2) // 2 + 2 * c["d"] * (c["d"] + 1) + 3
        return {"bytes": 8.0 * c["symbols"] * 8 + 16.0 * nf * nf, "flops": 4.0 * nf * nf * 2 * c["symbols"]}
    n = c["symbols"] * c["batch"]
    if kind == "ldbp":
        f = 8.0 * (2 * n * c["spans"] * c["steps"] * c["taps"] + n * c["mf_taps"])
        return {"bytes": 24.0 * n, "flops": (3 if c["train"] else 1) * f}
    f = sum(2.0 * 9 * i * o for i, o in CNN_LAYERS) * n
    return {"bytes": 16.0 * n, "flops": (3 if c["train"] else 1) * f}


# ---------------------------------------------------------------- 64-bit restatements
def _linear(spec, w2, hl):
    """exp(-alpha hl / 2) exp(i beta2 / 2 hl w^2) per realization (hl: tensor or number)."""
    hl = hl.view(-1, 1, 1) if isinstance(hl, torch.Tensor) else torch.full((1, 1, 1), hl, dtype=torch.float64, device=DEV)
    return spec * torch.polar(torch.exp(-0.5 * ALPHA * hl), (0.5 * BETA2 * hl) * w2)


def _ssfm64(x, dt, c, grid, steps, direction=1.0):
    """One span of the split step in 64 bits."""
    w2, kg, length = _omega2(x.shape[-1], dt), GAMMA * c.get("kappa", 1.0), c.get("span_m", 80e3)
    power = lambda a: (a.real * a.real + a.imag * a.imag).sum(1, keepdim=True)  # noqa: E731

    def kerr(spec, h):
        a = torch.fft.ifft(spec)
        p = power(a)
        h = h.view(-1, 1, 1) if isinstance(h, torch.Tensor) else h
        return torch.fft.fft(a * torch.polar(torch.ones_like(p), kg * h * p)), p

    if grid == "logarithmic":
        out = []
        for b in range(x.shape[0]):
            cl = c["phase"] / (GAMMA * float(power(x[b:b + 1]).mean())) / c["kappa"]
            eff = lambda d: (1 - math.exp(-ALPHA * d)) / ALPHA  # noqa: E731
            k = max(int(length / 1000.0), int(eff(length) / eff(cl)))
            g = (math.exp(-ALPHA * length) - 1) / k
            h = [-direction / ALPHA * math.log(1 + g / (1 + g * i)) for i in range(k)]
            out.append(_steps64(x[b:b + 1], w2, h, kerr))
        return torch.cat(out)
    if grid == "uniform":
        return _steps64(x, w2, [direction * length / steps] * steps, kerr)
    # phase-bounded steps, each realization on its own grid
    estimate = lambda p: torch.clamp(c["phase"] / (kg * p.amax((1, 2))), max=1000.0)  # noqa: E731
    h = estimate(power(x))
    done = torch.zeros_like(h)
    final = h >= length
    h = torch.where(final, torch.full_like(h, length), h)
    spec = _linear(torch.fft.fft(x), w2, 0.5 * direction * h)
    for i in range(100000):
        spec, p = kerr(spec, direction * h)
        done = done + h
        nxt = torch.where(final, torch.zeros_like(h), estimate(p))
        last = ~final & (done + nxt >= length)
        nxt = torch.where(last, length - done, nxt)
        spec = _linear(spec, w2, 0.5 * direction * (h + nxt))
        final, h = final | last, nxt
        if i % 16 == 15 and not bool((h > 0).any()):
            break
    return torch.fft.ifft(spec)


def _steps64(x, w2, h, kerr):
    spec = _linear(torch.fft.fft(x), w2, 0.5 * h[0])
    for i, s in enumerate(h):
        spec, _ = kerr(spec, s)
        spec = _linear(spec, w2, 0.5 * (s + (h[i + 1] if i + 1 < len(h) else 0.0)))
    return torch.fft.ifft(spec)


def _philox(seed, counter, streams, n):
    """Philox4x32-10 Gaussian pairs of counters {sample, stream, counter}, streams x n."""
    mask = 0xFFFFFFFF
    c = [torch.arange(n, device=DEV).expand(streams, n), torch.arange(streams, device=DEV).view(-1, 1).expand(streams, n),
         torch.full((streams, n), counter & mask, device=DEV), torch.full((streams, n), counter >> 32, device=DEV)]
    k0, k1 = seed & mask, (seed >> 32) & mask
    for _ in range(10):
        p0, p1 = c[0] * 0xD2511F53, c[2] * 0xCD9E8D57
        c = [((p1 >> 32) & mask) ^ c[1] ^ k0, p1 & mask, ((p0 >> 32) & mask) ^ c[3] ^ k1, p0 & mask]
        k0, k1 = (k0 + 0x9E3779B9) & mask, (k1 + 0xBB67AE85) & mask
    u1, u2 = ((c[0] >> 8).double() + 0.5) / 2 ** 24, (c[1] >> 8).double() / 2 ** 24
    return torch.polar(torch.sqrt(-2 * torch.log(u1)), 2 * math.pi * u2)


def _exact_fwd(c, seed):
    dt = 1 / (BAUD * c["osf"])
    x, g = _fwd_input(c, seed).to(C128), _gain(c)
    for span in range(c["spans"]):
        x = _ssfm64(x, dt, c, c["grid"], c.get("steps")) * math.sqrt(g)
        if c["nf_db"]:
            sigma = math.sqrt(PLANCK * F0 * 10 ** (c["nf_db"] / 10) * (g - 1) / 2 / dt / 2)
            x = x + sigma * _philox(seed, span, c["batch"] * c["modes"], c["samples"]).view_as(x)
    return x


def _exact_dbp(c, seed):
    out = []
    xs = [x.to(C128) for x in _dbp_inputs(c, seed)]
    for k in _dbp_steps(c):
        for x in xs:
            for _ in range(c["spans"]):
                x = _ssfm64(x / math.sqrt(_gain(c)), 1 / (2 * BAUD), c, "uniform", k, -1.0)
            out.append(x)
    return out


def _rrc_filter(x, osf):
    h = torch.as_tensor(np.fft.ifftshift(_rrc_pulse(x.shape[-1] // osf, osf, ROLL_OFF)), device=DEV)
    return torch.fft.ifft(torch.fft.fft(x) * torch.fft.fft(h)) / x.shape[-1]


def _shift(x, turns):
    """x exp(2 pi i turns n)"""
    n = torch.arange(x.shape[-1], device=DEV, dtype=torch.float64)
    return x * torch.polar(torch.ones_like(n), 2 * math.pi * torch.remainder(turns * n, 1.0))


GRAY = np.array([complex(re, im) for im in (-3, -1, 3, 1) for re in (-3, -1, 3, 1)]) / math.sqrt(10.0)


def _exact_tx(c, seed):
    codes = np.random.default_rng(seed).integers(0, 16, (c["channels"], c["modes"], c["symbols"]))
    x = torch.zeros(c["channels"], c["modes"], c["symbols"] * c["osf"], dtype=C128, device=DEV)
    x[..., ::c["osf"]] = torch.as_tensor(GRAY[codes] * math.sqrt(_watts(0.0) / c["modes"]), device=DEV)
    x = _rrc_filter(x, c["osf"]) * c["osf"]
    dt = 1 / (BAUD * c["osf"])
    return sum(_shift(x[i], (i - c["channels"] // 2) * SPACING * dt) for i in range(c["channels"]))[None]


def _exact_rx(c, seed):
    x, t = (v.to(C128) for v in _rx_input(c, seed))
    n, m, dt = x.shape[-1], 2 * c["symbols"], 1 / (BAUD * c["osf"])
    s = torch.fft.fft(x)
    cut = int(0.5 * SPACING * (n * dt)) + 1
    s[..., cut:n - cut + 1] = 0
    s = torch.cat([s[..., :m // 2], s[..., n - m // 2:]], -1)
    s = s * torch.polar(torch.ones((), dtype=torch.float64, device=DEV),
                        -0.5 * BETA2 * 80e3 * c["spans"] * _omega2(m, 1 / (2 * BAUD)))
    y = _rrc_filter(torch.fft.ifft(s) * m / n, 2)[..., ::2]
    a = 2 * math.pi * torch.arange(720, device=DEV, dtype=torch.float64) / 720
    z = (t.conj() * y).sum((1, 2)).view(-1, 1)
    best = a[(z.real * torch.cos(a) - z.imag * torch.sin(a)).argmax(1)].view(-1, 1, 1)
    return y * torch.polar(torch.ones_like(best), best)


def _exact_decide(c, seed):
    t, r = (v.to(C128) for v in _noisy_symbols(c, seed, c["batch"], c["modes"], 0.2))
    pts = torch.as_tensor(GRAY, device=DEV)
    mean = lambda v: (v.abs() ** 2).mean((1, 2), keepdim=True).sqrt()  # noqa: E731
    code = lambda v, s: ((v / s)[..., None] - pts).abs().argmin(-1)  # noqa: E731
    codes = code(r, mean(r))
    bits = code(t, mean(t)) ^ code(r, mean(t))
    count = sum((bits >> i) & 1 for i in range(4)).sum((1, 2)).double()
    q2 = -10 * torch.log10(((t - r).abs() ** 2).sum((1, 2)) / (t.abs() ** 2).sum((1, 2)))
    return {"hard": pts[codes] * mean(r), "codes": codes.to(torch.int32), "ber": count / (4.0 * c["modes"] * c["symbols"]),
            "q2": q2}


def _at(x, d):
    """x[k + d], zero outside the realization."""
    out = torch.zeros_like(x)
    n = x.shape[-1]
    if d >= 0:
        out[..., :max(0, n - d)] = x[..., d:]
    else:
        out[..., -d:] = x[..., :n + d]
    return out


def _triplets64(x, w):
    """sum over (m, n) of w[R+m, R+n] x_p[k+m] sum_q x_q[k+n] conj(x_q[k+m+n]), zero in the
    first and last R samples; x: batch x modes x samples."""
    r = (w.shape[0] - 1) // 2
    n = x.shape[-1]
    size = 1 << (n + 4 * r + 2).bit_length()
    w = torch.as_tensor(w, device=DEV)
    out = torch.zeros_like(x)
    ext = torch.nn.functional.pad(x, (2 * r, 2 * r))  # sample k at index k + 2r
    for m in range(-r, r + 1):
        row = w[r + m]
        if not bool((row != 0).any()):
            continue
        q = (ext * _at(ext, m).conj()).sum(1)
        # s[k] = sum_n row[n] q[k + n]: a circular correlation, long enough not to wrap
        kern = torch.zeros(size, dtype=C128, device=DEV)
        kern[torch.arange(-r, r + 1, device=DEV) % size] = row.flip(0)
        s = torch.fft.ifft(torch.fft.fft(q, size) * torch.fft.fft(kern))[..., 2 * r:2 * r + n]
        out += _at(x, m) * s[:, None]
    out[..., :r] = 0
    out[..., n - r:] = 0
    return out


def _dense(radius, m, n, k):
    w = np.zeros((2 * radius + 1, 2 * radius + 1), complex)
    w[radius + m, radius + n] = k
    return w


def _diamond(w):
    r = (w.shape[0] - 1) // 2
    a = np.abs(np.arange(-r, r + 1))
    return np.where(a[:, None] + a[None, :] <= r, w, 0)


def _neighbours(x, pol, m, n):
    """Cross-phase triplet T1(m, n) + T3(m, -n) of polarization `pol` (rows:
    left neighbour 0-1, centre 2-3, right neighbour 4-5)."""
    out = 0
    for lo, nn in ((0, n), (4, -n)):
        p, q = x[:, lo + pol], x[:, lo + 1 - pol]
        same = 2 * _at(p, nn) * _at(p, m + nn).conj() + _at(q, nn) * _at(q, m + nn).conj()
        out = out + _at(x[:, 2 + pol], m) * same + _at(x[:, 3 - pol], m) * (_at(p, nn) * _at(q, m + nn).conj())
    return out


def _exact_ppe_wdm(c, seed):
    x, r = (v.to(C128) for v in _noisy_symbols(c, seed, c["batch"], 6, 0.1))
    y = _triplets64(x[:, 2:4], _diamond(_table(seed, c["c"], 4e-3)))
    w, d = _table(seed + 1, c["d"], 4e-3), c["d"]
    z = torch.zeros_like(y)
    for m in range(-d, d + 1):
        for n in range(-(d - abs(m)), d - abs(m) + 1):
            z += complex(w[d + m, d + n]) * torch.stack([_neighbours(x, 0, m, n), _neighbours(x, 1, m, n)], 1)
    z[..., :d] = 0
    z[..., c["symbols"] - d:] = 0
    return (r[:, 2:4] - y - z) / (0.98 + 0.05j)


def _exact_fit(c, seed):
    x, r = (v.to(C128) for v in _noisy_symbols(c, seed, 1, 6, 0.1))
    cr, d, big = c["c"], c["d"], max(c["c"], c["d"])
    centre, cols, images = x[:, 2:4], [], []
    term = lambda m, n: _at(centre, m) * (_at(centre, n) * _at(centre, m + n).conj()).sum(1, keepdim=True)  # noqa: E731
    for m in range(-(cr // 2), cr // 2 + 1):
        for n in range(abs(m), cr - abs(m) + 1):
            im = sorted({(m, n), (n, m), (-m, -n), (-n, -m)})
            cols.append(sum(term(a, b) for a, b in im))
            images.append(im)
    cross = [(m, n) for m in range(-d, d + 1) for n in range(-(d - abs(m)), d - abs(m) + 1)]
    cols += [torch.stack([_neighbours(x, 0, m, n), _neighbours(x, 1, m, n)], 1) for m, n in cross] + [centre]
    cut = slice(big, c["symbols"] - big)
    a = torch.stack([v[0][:, cut].reshape(-1) for v in cols], 1)
    y = r[0, 2:4][:, cut].reshape(-1)
    a, y = a - a.mean(0), y - y.mean()
    size = a.abs().square().mean(0).sqrt()
    q, up = torch.linalg.qr(a / size)
    w = (torch.linalg.solve_triangular(up, (q.conj().T @ y)[:, None], upper=True)[:, 0] / size).cpu().numpy()
    tc, td = np.zeros((2 * cr + 1, 2 * cr + 1), complex), np.zeros((2 * d + 1, 2 * d + 1), complex)
    for i, im in enumerate(images):
        for m, n in im:
            tc[cr + m, cr + n] = w[i]
    for i, (m, n) in enumerate(cross):
        td[d + m, d + n] = w[len(images) + i]
    return {"C": tc, "D": td, "linear": np.complex128(w[-1])}


def _exact_ldbp(c, seed):
    x, t = (v.to(C128) for v in _ldbp_input(c, seed))
    h, xi, hmf = (torch.as_tensor(v, device=DEV) for v in _ldbp_params(c))
    h, hmf, xi = h.to(C128).requires_grad_(c["train"]), hmf.to(C128).requires_grad_(c["train"]), xi.double().requires_grad_(c["train"])
    n = x.shape[-1]

    def fir(x, h):
        half = (h.numel() - 1) // 2
        pad = torch.zeros(n, dtype=C128, device=DEV).index_put((torch.arange(-half, half + 1, device=DEV) % n,), h)
        return torch.fft.ifft(torch.fft.fft(x) * (torch.fft.ifft(pad) * n))

    def step(x, h, k, scale):
        y = fir(x * scale, h)
        p = y.real * y.real + y.imag * y.imag
        return y * torch.polar(torch.ones_like(p), k * p)

    scale = float(np.float32(_gain(c) ** -0.5))
    with torch.set_grad_enabled(c["train"]):
        for i in range(c["spans"] * c["steps"]):
            x = step(x, h[i], xi[i], scale if i % c["steps"] == 0 else 1.0)
        y = fir(x, hmf)[..., ::2]
        if not c["train"]:
            return y
        loss = (y - t).abs().square().mean()
        loss.backward()
    # torch's complex gradient is twice the derivative to the conjugate
    return {"loss": float(loss), "h": h.grad / 2, "xi": xi.grad, "hmf": hmf.grad / 2}


def _exact_cnn(c, seed):
    t, y = (v.to(C128)[:, 0] for v in _noisy_symbols(c, seed, c["batch"], 1, 0.1))
    flat = torch.as_tensor(_cnn_params(seed), device=DEV).double().requires_grad_(c["train"])
    feats = [y]
    for m, n in CNN_TRIPLETS:
        f = _at(y, m) * _at(y, n) * _at(y, m + n).conj()
        feats.append(f if (m, n) == (0, 0) else f + _at(y, -m) * _at(y, -n) * _at(y, -m - n).conj())
    x = torch.view_as_real(torch.stack(feats, 1)).permute(0, 1, 3, 2).reshape(y.shape[0], 16, -1)
    with torch.set_grad_enabled(c["train"]):
        o = 0
        for i, (cin, cout) in enumerate(CNN_LAYERS):
            w = flat[o:o + cout * 9 * cin].view(cout, 9, cin)
            o += cout * 9 * cin
            b = flat[o:o + cout]
            o += cout
            # nine products instead of a convolution call: 64-bit ones are slow there
            p = torch.nn.functional.pad(x, (4, 4))
            x = sum(torch.einsum("oi,bil->bol", w[:, k], p[..., k:k + y.shape[1]]) for k in range(9)) + b[:, None]
            x = torch.relu(x) if i < 3 else x
        z = y + torch.complex(x[:, 0], x[:, 1])
        if not c["train"]:
            return z[:, None]
        loss = (z - t).abs().square().mean()
        loss.backward()
    return {"loss": float(loss), "grads": flat.grad}


def exact(case, seed):
    c = case
    with torch.no_grad():
        kind = c["kind"]
        if kind == "fwd":
            return _exact_fwd(c, seed)
        if kind == "dbp":
            return _exact_dbp(c, seed)
        if kind == "tx":
            return _exact_tx(c, seed)
        if kind == "rx":
            return _exact_rx(c, seed)
        if kind == "decide":
            return _exact_decide(c, seed)
        if kind == "ppe":
            t, _ = _noisy_symbols(c, seed, 1, c["modes"], 0.1)
            return _triplets64((t * math.sqrt(0.5)).to(C128), _dense(c["radius"], *_ppe_terms(c, seed)))
        if kind == "ppe_wdm":
            return _exact_ppe_wdm(c, seed)
        if kind == "ppe_fit":
            return _exact_fit(c, seed)
    return _exact_ldbp(c, seed) if c["kind"] == "ldbp" else _exact_cnn(c, seed)
