"""What this framework's speed is measured on: the calls its users make, through the public
entry points, at the sizes of the scripts, the benchmark and the tests.

Every case is a dict of plain values with a ``kind``:

  step       real_field.rk2_step_table with inline hash noise (a caller's own loop)
  script     one step of the real command's default loop: noise field, table step with that
             field and the folded range, range read on the host
  thermal    real_field.rk2_fused_single_pass (the command's rk2_fused_inline): the one-loop
             V' evaluated per site
  driver     driver.Simulation.run: a graph-captured chunk with the observables of every step
  cstep      complex_field.rk2_step_table with inline hash noise and the eps term
  cscript    one step of the complex command's RK2 loop, as ``script``
  integrator the first-order and BAOAB steps of both fields
  winding    complex_field.compute_winding_number
  label      labels.label of the bubbles of a field
  ensemble   ensemble.Ensemble.run over mixed replicas
  train      one SurrogateNet training step (gradient and Adam)

A state is what a program holds between calls; the steppers advance it, with the step number
as the noise counter, so a second call is the program's next step.
"""
import math

import numpy as np
import torch

from thermal_inflation_phase_transition_b200 import complex_field as CF
from thermal_inflation_phase_transition_b200 import driver as D
from thermal_inflation_phase_transition_b200 import ensemble as EN
from thermal_inflation_phase_transition_b200 import labels as LB
from thermal_inflation_phase_transition_b200 import real_field as RF
from thermal_inflation_phase_transition_b200.surrogate import SurrogateNet
from thermal_inflation_phase_transition_b200.thermal import ThermalPotential

DEV = "cuda"

# ------------------------------------------------------------------- cases ---


def listed():
    return [
        # the 2-D lattice in FP64: the smallest call, where the launch and the host count
        dict(name="step_2d_256_f64", kind="step", storage="f64", nx=256, ny=256, nz=1, table="1d",
             ranged=False),
        # the headline lattice in compensated FP32 with the (phi, T) table
        dict(name="step_512_f32c", kind="step", storage="f32c", nx=512, ny=512, nz=512,
             table="2d", ranged=False),
        # the real command as it runs without options: 256^3, float32, 16384-point table
        dict(name="script_256_f32", kind="script", storage="f32", nx=256, ny=256, nz=256),
        # the real command's long production runs: inline thermal V', inline noise
        dict(name="thermal_256_f32", kind="thermal", storage="f32", nx=256, ny=256, nz=256),
        # a run of the graph-captured driver on a lattice of odd extents in FP64
        dict(name="driver_odd_f64", kind="driver", storage="f64", nx=126, ny=131, nz=98, steps=20),
        # the complex field in compensated FP32
        dict(name="cstep_256_f32c", kind="cstep", storage="f32c", nx=256, ny=256, nz=256),
        # the complex command's RK2 loop on the flat production lattice
        dict(name="cscript_512x512x64_f32", kind="cscript", storage="f32", nx=512, ny=512, nz=64,
             zn=0),
        # the complex command without options takes the first-order integrator
        dict(name="overdamped_complex_256_f32", kind="integrator", method="overdamped",
             field="complex", storage="f32", nx=256, ny=256, nz=256),
        # winding numbers of a string network, as every complex snapshot needs them
        dict(name="winding_256_f32", kind="winding", storage="f32", nx=256, ny=256, nz=256),
        # bubbles of a snapshot, ragged extents
        dict(name="label_250_f32", kind="label", storage="f32", nx=250, ny=243, nz=237, level=1.0),
        # two check intervals of the batched ensemble: 2-D, 64^3 and 96^3 replicas
        dict(name="ensemble_112", kind="ensemble", n2d=64, l2d=128, na=32, la=64, nb=16, lb=96,
             steps=20),
        # one training step of the surrogate at its default batch
        dict(name="train_4096", kind="train", rows=4096),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _box(rng, lo, hi, most):
    """Three extents in [lo, hi] with at most `most` sites: cubes, flat boxes and odd ones."""
    while True:
        a = _log(rng, lo, hi)
        form = rng.choice(("cube", "flat", "odd", "odd"))
        if form == "cube":
            a = max(8, a // 8 * 8)
            s = (a, a, a)
        elif form == "flat":
            a = max(8, a // 8 * 8)
            s = (a, a, max(4, a // 8 // 4 * 4))
        else:
            s = tuple(max(4, int(a * rng.uniform(0.7, 1.4))) for _ in range(3))
        if s[0] * s[1] * s[2] <= most:
            return dict(nx=s[0], ny=s[1], nz=s[2])


def draw(rng):
    kind = rng.choice(("step", "step", "script", "thermal", "driver", "cstep", "cscript",
                       "integrator", "winding", "label", "ensemble", "train"))
    st = rng.choice(("f32c", "f32", "f64"))
    if kind == "step":
        if rng.random() < 0.25:
            size = dict(nx=_log(rng, 64, 2048), ny=_log(rng, 64, 2048), nz=1)
        else:
            size = _box(rng, 24, 512, 1 << 27)
        return dict(kind=kind, storage=st, table=rng.choice(("1d", "2d")),
                    ranged=rng.random() < 0.5, **size)
    if kind in ("script", "thermal"):
        return dict(kind=kind, storage=st, **_box(rng, 32, 320, 1 << 24))
    if kind == "driver":
        return dict(kind=kind, storage=st, steps=rng.choice((10, 20, 50)),
                    **_box(rng, 32, 200, 1 << 22))
    if kind == "cstep":
        return dict(kind=kind, storage=st, **_box(rng, 32, 384, 1 << 25))
    if kind == "cscript":
        return dict(kind=kind, storage=st, zn=rng.choice((0, 0, 4)),
                    **_box(rng, 32, 320, 1 << 24))
    if kind == "integrator":
        return dict(kind=kind, storage=st, method=rng.choice(("overdamped", "baoab")),
                    field=rng.choice(("real", "complex")), **_box(rng, 32, 320, 1 << 24))
    if kind == "winding":
        return dict(kind=kind, storage=st, **_box(rng, 24, 400, 1 << 25))
    if kind == "label":
        return dict(kind=kind, storage=st, level=rng.uniform(0.3, 2.0),
                    **_box(rng, 24, 400, 1 << 25))
    if kind == "ensemble":
        return dict(kind=kind, n2d=rng.randint(1, 64), l2d=_log(rng, 48, 160),
                    na=rng.randint(1, 30), la=rng.choice((32, 48, 50, 64)),
                    nb=rng.randint(1, 15), lb=rng.choice((66, 80, 96)), steps=20)
    return dict(kind="train", rows=_log(rng, 100, 20000))


def _sites(c):
    return c["nx"] * c["ny"] * c["nz"]


def work(case):
    """Bytes: the inputs read once and the outputs written once (per step where a call makes
    several).  flops: the arithmetic of the update written out (stencil, V', noise)."""
    k = case["kind"]
    if k == "train":
        p, r = 6 * 128 + 2 * 128 * 128 + 128 * 17, case["rows"]
        return {"bytes": 4.0 * (39328 * 7 + r * 26), "flops": 6.0 * p * r}
    if k == "ensemble":
        n = case["n2d"] * case["l2d"] ** 2 + case["na"] * case["la"] ** 3 + case["nb"] * case["lb"] ** 3
        return {"bytes": 32.0 * n * case["steps"], "flops": 100.0 * n * case["steps"]}
    n, v = _sites(case), {"f32": 4, "f64": 8, "f32c": 8}[case["storage"]]
    a = 4 if case["storage"] == "f32" else 8      # an element of a noise array
    if k == "step":
        return {"bytes": 4.0 * v * n, "flops": 100.0 * n}
    if k == "script":
        return {"bytes": (4.0 * v + a) * n, "flops": 100.0 * n}
    if k == "thermal":
        return {"bytes": 4.0 * v * n, "flops": 400.0 * n}
    if k == "driver":
        return {"bytes": 4.0 * v * n * case["steps"], "flops": 120.0 * n * case["steps"]}
    if k == "cstep":
        return {"bytes": 8.0 * v * n, "flops": 200.0 * n}
    if k == "cscript":
        return {"bytes": (8.0 * v + 2 * a) * n, "flops": 200.0 * n}
    if k == "integrator":
        f = (1 if case["field"] == "real" else 2) * (2 if case["method"] == "baoab" else 1)
        return {"bytes": 2.0 * v * f * n, "flops": 60.0 * f * n}
    if k == "winding":
        return {"bytes": (2.0 * v + 4) * n, "flops": 40.0 * n}
    return {"bytes": (v + 4.0) * n, "flops": 10.0 * n}          # label


# ------------------------------------------------------------------ inputs ---
# the lattice model of the benchmark: V = D (T^2 - T0^2) phi^2 - E T phi^3 + lam/4 phi^4
DT, DX, ETA, T_TOY, NPHI, LO, HI = 0.05, 1.0, 1.0, 0.98, 4096, 0.0, 3.0
NT_TAB, T_LO, T_HI = 256, 0.97, 1.06
EPS4 = 1e-3
# the scripts' units (GeV): couplings, temperature, steps
MPHI, T_PHYS, DX_PHYS = 1000.0, 7350.0, 1e-3
COUPLINGS = (1.0e6, 1.09, 1.05, 1.09, 1.05)   # boson mass^2, gb, gb gauge, gf, gf gauge
LAM_REAL, LAM_CPLX = 1e-24, 1e-16
COEF_REAL, COEF_CPLX = (20.0, 20.0), (2.0, -1.0)
DT_SCRIPT, ETA_REAL, ETA_CPLX = 0.1, T_PHYS / MPHI, 1.0
TABLE_SIZE = 16384                             # the scripts' table


def _toy_vprime(x, T):
    return 2.0 * 0.1 * (T * T - 1.0) * x - 3.0 * 0.05 * T * x * x + 0.1 * x * x * x


def _toy_ns(T=T_TOY):
    return math.sqrt(2.0 * ETA * T * DT)


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _randn(shape, g, scale, mean=0.0):
    return torch.randn(shape, dtype=torch.float64, device=DEV, generator=g).mul_(scale).add_(mean)


def _as(x, storage):
    """A float64 field in the storage, and the float64 value that the storage holds."""
    if storage == "f64":
        return x
    if storage == "f32":
        return x.float()
    hi = x.float()
    return torch.stack([hi, (x - hi.double()).float()])


def _value(t):
    return t[0].double() + t[1].double() if t.dim() == 4 else t.double()


def _shape(c):
    return (c["nx"], c["ny"], c["nz"])


def _toy_table(two_d):
    x = np.linspace(LO, HI, NPHI)
    dinv = 1.0 / ((HI - LO) / (NPHI - 1))
    if not two_d:
        return torch.from_numpy(_toy_vprime(x, T_TOY)).to(DEV), dinv
    Ts = np.linspace(T_LO, T_HI, NT_TAB)
    return torch.from_numpy(np.stack([_toy_vprime(x, t) for t in Ts])).to(DEV), dinv


def _toy_state(case, seed, complex_):
    """Fields in the thermal spread that the toy model's runs settle into."""
    g, sh = _gen(seed), _shape(case)
    if complex_:
        f = [_randn(sh, g, 0.5, 0.2), _randn(sh, g, 0.5), _randn(sh, g, 1.0), _randn(sh, g, 1.0)]
    else:
        f = [_randn(sh, g, 0.5, 0.4), _randn(sh, g, 1.0)]
    return [_as(x, case["storage"]) for x in f]


def _script_state(case, seed, complex_):
    """Fields in the scripts' units at their starting temperature."""
    g, sh = _gen(seed), _shape(case)
    n = 2 if complex_ else 1
    f = [_randn(sh, g, 1350.0) for _ in range(n)] + [_randn(sh, g, 2711.0) for _ in range(n)]
    return [_as(x, case["storage"]) for x in f]


def _potential(complex_):
    return ThermalPotential(lam=LAM_CPLX if complex_ else LAM_REAL, mphi=MPHI,
                            pot_coeffs=COEF_CPLX if complex_ else COEF_REAL, device=DEV)


def _table_bounds(fields, complex_):
    """The commands' table range: the field's own plus a margin of at least 20000."""
    if complex_:
        hi = float(torch.sqrt(_value(fields[0]) ** 2 + _value(fields[1]) ** 2).max())
        return 0.0, hi + max(max(hi, 1.0), 20000.0)
    v = _value(fields[0])
    lo, hi = float(v.min()), float(v.max())
    m = max(max(hi - lo, 1.0), 20000.0)
    return lo - m, hi + m


def _noise_dtype(storage):
    return torch.float32 if storage == "f32" else torch.float64


def _smooth(shape, g, passes):
    x = torch.randn(shape, dtype=torch.float64, device=DEV, generator=g)
    for _ in range(passes):
        for d in range(3):
            if shape[d] > 1:
                x = (x + x.roll(1, d) + x.roll(-1, d)) / 3.0
    return x / x.std()


def _specs(case, seed):
    r = np.random.default_rng(1000 + int(seed))
    shapes = ([(case["l2d"], case["l2d"], 1)] * case["n2d"] + [(case["la"],) * 3] * case["na"]
              + [(case["lb"],) * 3] * case["nb"])
    T, E = r.uniform(0.98, 1.01, len(shapes)), r.uniform(0.04, 0.06, len(shapes))
    return [(s, float(t), float(e), 1000 * int(seed) + q)
            for q, (s, t, e) in enumerate(zip(shapes, T, E))]


def _train_rows(case, seed):
    """Normalised parameters, and targets as the ensemble engine's replicas give them: event,
    exposure, the two weights, the converted fraction at 16 times."""
    r = np.random.default_rng(50 + int(seed))
    n = case["rows"]
    x = r.uniform(-1.0, 1.0, (n, 6)).astype(np.float32)
    t = np.zeros((n, 20), np.float32)
    t[:, 0] = r.random(n) < 0.4
    t[:, 1] = r.exponential(1.0, n)
    t[:, 2] = 1.0
    t[:, 3] = 1.0
    t[:, 4:] = np.sort(np.clip(r.normal(0.3, 0.4, (n, 16)), 0.0, 1.0), axis=1)
    w = r.normal(0.0, 1.0, 39328)
    return x, t, w


MLP_DIMS = (16, 128, 128, 128, 32)


def _mlp_params(w):
    """He-normal weights on the live rows and columns, zero padding, small biases."""
    p, off = np.zeros(39328, np.float32), 0
    for li in range(4):
        fi, fo = MLP_DIMS[li], MLP_DIMS[li + 1]
        rows, cols = (6 if li == 0 else fi), (17 if li == 3 else fo)
        s = math.sqrt(2.0 / rows) if li < 3 else 0.1 / math.sqrt(rows)
        W = np.zeros((fi, fo))
        W[:rows, :cols] = w[off:off + fi * fo].reshape(fi, fo)[:rows, :cols] * s
        p[off:off + fi * fo] = W.reshape(-1)
        b = np.zeros(fo)
        b[:cols] = 0.01 * w[off + fi * fo:off + fi * fo + cols]
        p[off + fi * fo:off + fi * fo + fo] = b
        off += fi * fo + fo
    return p


# ----------------------------------------------------------------- prepare ---
def prepare(case, seed):
    k = case["kind"]
    s = dict(case=case, n=int(seed) + 3, seed=int(seed))
    if k in ("step", "cstep"):
        f = _toy_state(case, seed, k == "cstep")
        s.update(f=f, tmp=[torch.empty_like(x) for x in f])
        s["tab"], s["dinv"] = _toy_table(case.get("table") == "2d")
        s["range"] = RF.PhiRange(DEV) if case.get("ranged") else None
    elif k in ("script", "cscript"):
        c = k == "cscript"
        f = _script_state(case, seed, c)
        s.update(f=f, tmp=[torch.empty_like(x) for x in f], tp=_potential(c), range=RF.PhiRange(DEV))
        s["noise"] = [torch.empty(_shape(case), dtype=_noise_dtype(case["storage"]), device=DEV)
                      for _ in range(2 if c else 1)]
        s["tab"] = s["tp"].table(T_PHYS, *_table_bounds(f, c), TABLE_SIZE)
    elif k == "thermal":
        f = _script_state(case, seed, False)
        s.update(f=f, tmp=[torch.empty_like(x) for x in f], tp=_potential(False))
    elif k == "driver":
        g, sh = _gen(seed), _shape(case)
        phi0, pi0 = _randn(sh, g, 0.5, 0.4), _randn(sh, g, 1.0)
        s["sim"] = D.Simulation(sh, storage=case["storage"], dt=DT, dx=DX, eta=ETA,
                                table=D.Table2D.build(_toy_vprime, LO, HI, NPHI, T_LO, T_HI, NT_TAB),
                                schedule=D.linear_cooling(1.0, 0.98, 4000, 4000, dt=DT),
                                seed=s["seed"], phi0=phi0.cpu().numpy(), pi0=pi0.cpu().numpy(),
                                graph_steps=case["steps"], device=DEV)
    elif k == "integrator":
        c = case["field"] == "complex"
        f = _script_state(case, seed, c)
        if case["method"] == "overdamped":
            f = f[:2 if c else 1]
        s.update(f=f, tmp=[torch.empty_like(x) for x in f], tp=_potential(c))
        s["tab"] = s["tp"].table(T_PHYS, *_table_bounds(f, c), TABLE_SIZE)
    elif k == "winding":
        g = _gen(seed)
        s["f"] = [_as(_smooth(_shape(case), g, 3), case["storage"]) for _ in range(2)]
        s["out"] = torch.empty(_shape(case), dtype=torch.float32, device=DEV)
    elif k == "label":
        s["f"] = _as(_smooth(_shape(case), _gen(seed), 4), case["storage"])
    elif k == "ensemble":
        # retire_frac = 1 keeps every replica stepping (its conversion curve runs on)
        s["ens"] = EN.Ensemble([EN.ReplicaSpec(*a) for a in _specs(case, seed)], storage="f32c",
                               check_every=10, retire_frac=1.0, init_seed=s["seed"], device=DEV)
    else:
        x, t, w = _train_rows(case, seed)
        s["net"] = SurrogateNet(_mlp_params(w), device=DEV)
        s["x"], s["t"] = torch.from_numpy(x).to(DEV), torch.from_numpy(t).to(DEV)
    return s


# --------------------------------------------------------------------- run ---
def _read_range(r):
    lo, hi, bad = RF.PhiRange.decode(r.last.cpu().numpy())
    return [lo, hi, float(bad)]


def _script_ns(eta):
    return math.sqrt(2.0 * eta * T_PHYS * DT_SCRIPT / (MPHI ** 2 * DX_PHYS ** 3))


def run(s):
    case = s["case"]
    k = case["kind"]
    n = s["n"]
    s["n"] = n + 1
    if k == "step":
        kw = dict(vp_T=T_TOY, vp_T_min=T_LO, vp_T_dinv=1.0 / ((T_HI - T_LO) / (NT_TAB - 1))) \
            if case["table"] == "2d" else {}
        RF.rk2_step_table(s["f"][0], s["f"][1], DT, DX, ETA, 1.0, None, s["tmp"][0], s["tmp"][1],
                          1.0, s["tab"], LO, s["dinv"], NPHI, noise_scale=_toy_ns(), noise_step=n,
                          seed=s["seed"], phi_range=s["range"], **kw)
        return s["f"]
    if k == "cstep":
        CF.rk2_step_table(*s["f"], DT, DX, ETA, 1.0, None, None, *s["tmp"], 1.0, s["tab"], LO,
                          s["dinv"], NPHI, eps4=EPS4, noise_scale=_toy_ns(), noise_step=n,
                          seed=s["seed"])
        return s["f"]
    if k == "script":
        RF.generate_noise_field(s["noise"][0], _script_ns(ETA_REAL), n)
        RF.rk2_step_table(s["f"][0], s["f"][1], DT_SCRIPT, 1.0, ETA_REAL, MPHI, s["noise"][0],
                          s["tmp"][0], s["tmp"][1], 1.0, *s["tab"], TABLE_SIZE,
                          phi_range=s["range"])
        return s["f"] + s["noise"] + _read_range(s["range"])
    if k == "cscript":
        for c in range(2):
            RF.generate_noise_field(s["noise"][c], _script_ns(ETA_CPLX), n, component=c)
        zn = (4.0, 1e10, 1.0) if case["zn"] else (0.0, 0.0, 0.0)
        CF.rk2_step_table(*s["f"], DT_SCRIPT, 1.0, ETA_CPLX, MPHI, *s["noise"], *s["tmp"], 1.0,
                          *s["tab"], TABLE_SIZE, zn=zn, rho_range=s["range"])
        return s["f"] + s["noise"] + _read_range(s["range"])
    if k == "thermal":
        RF.rk2_fused_single_pass(s["f"][0], s["f"][1], DT_SCRIPT, 1.0, ETA_REAL, T_PHYS,
                                 T_PHYS * (1 - 1e-6), MPHI, LAM_REAL, MPHI, *COUPLINGS,
                                 _script_ns(ETA_REAL), n, s["tmp"][0], s["tmp"][1], 1.0,
                                 splines=s["tp"])
        return s["f"]
    if k == "driver":
        obs = s["sim"].run(case["steps"])
        return [obs, s["sim"].phi[0], s["sim"].pi[0]]
    if k == "integrator":
        args = (DT_SCRIPT, 1.0, _integrator_eta(case), MPHI, 1.0, *s["tab"], TABLE_SIZE,
                _integrator_ns(case), n)
        if case["field"] == "real":
            if case["method"] == "overdamped":
                RF.overdamped_euler_step_table(s["f"][0], *args, phi_tmp=s["tmp"][0])
            else:
                RF.baoab_step_table(*s["f"], *args, phi_tmp=s["tmp"][0], pi_tmp=s["tmp"][1])
        elif case["method"] == "overdamped":
            CF.overdamped_euler_step_table(*s["f"], *args, tmp=s["tmp"])
        else:
            CF.baoab_step_table(*s["f"], *args, tmp=s["tmp"])
        return s["f"]
    if k == "winding":
        return CF.compute_winding_number(s["f"][0], s["f"][1], s["out"])
    if k == "label":
        return list(LB.label(s["f"], case["level"]))
    if k == "ensemble":
        e = s["ens"]
        first = e.run(e.steps_done + case["steps"], record_curves=False)
        return [first, e.frac, e.phi[0], e.pi[0]]
    g = s["net"].grad(s["x"], s["t"])
    s["net"].adam(g, 2e-3)
    return [g, s["net"].params]


def _integrator_eta(case):
    return ETA_REAL if case["field"] == "real" else ETA_CPLX


def _integrator_ns(case):
    q = MPHI ** 2 * DX_PHYS ** 3
    if case["method"] == "overdamped":
        return math.sqrt(2.0 * T_PHYS * DT_SCRIPT / (_integrator_eta(case) * q))
    return math.sqrt(T_PHYS / q)


# ------------------------------------------------------------------- exact ---
# The same steps in float64 torch and numpy, written from the definitions alone.
_M64 = (1 << 64) - 1


def _s64(c):
    c &= _M64
    return c - (1 << 64) if c >> 63 else c


def _shr(x, k):
    return (x >> k) & ((1 << (64 - k)) - 1)


def _uniforms(n_sites, step, mul, seed, first=0):
    x = torch.arange(first, first + n_sites, dtype=torch.int64, device=DEV) * mul
    x = (x ^ _s64(step)) + _s64(seed * 0x9E3779B97F4A7C15)
    x = (x ^ _shr(x, 30)) * _s64(0xBF58476D1CE4E5B9)
    x = (x ^ _shr(x, 27)) * _s64(0x94D049BB133111EB)
    x = x ^ _shr(x, 31)
    u1 = _shr(x, 11).double() * 2.0 ** -53
    x = (x * _s64(0x2545F4914F6CDD1D)) ^ _s64(0x9E3779B97F4A7C15)
    x = (x ^ _shr(x, 30)) * _s64(0xBF58476D1CE4E5B9)
    x = x ^ _shr(x, 31)
    return u1.clamp_(min=1e-12), _shr(x, 11).double() * 2.0 ** -53


def _normals(shape, step, mul, seed, both=False):
    n = int(np.prod(shape))
    z1 = torch.empty(n, dtype=torch.float64, device=DEV)
    z2 = torch.empty_like(z1) if both else None
    b = 1 << 24
    for o in range(0, n, b):
        m = min(b, n - o)
        u1, u2 = _uniforms(m, step, mul, seed, o)
        r, a = torch.sqrt(-2.0 * torch.log(u1)), 6.283185307179586 * u2
        z1[o:o + m] = r * torch.cos(a)
        if both:
            z2[o:o + m] = r * torch.sin(a)
    return (z1.view(shape), z2.view(shape)) if both else z1.view(shape)


PASS2, PASS4 = 73856093, 19349669


def _lap(a):
    out = a * -6.0
    for d in range(3):
        out += a.roll(1, d)
        out += a.roll(-1, d)
    return out


def _lerp(t, lo, dinv, x):
    f = (x - lo) * dinv
    i = f.clamp(0.0, float(t.numel() - 2)).long()
    a = t[i]
    return a + (f - i) * (t[i + 1] - a)


def _toy_vp(two_d, T=T_TOY):
    """The lookup in the toy table, its row blended at T for the 2-D one."""
    t, dinv = _toy_table(two_d)
    if two_d:
        ft = (T - T_LO) * (1.0 / ((T_HI - T_LO) / (NT_TAB - 1)))
        i = min(max(int(ft), 0), NT_TAB - 2)
        t = t[i] + (ft - i) * (t[i + 1] - t[i])
    return lambda x: _lerp(t, LO, dinv, x)


_DJ = {}


def _dj_spline(fermion):
    """Not-a-knot cubic of dJ(u) = int_0^100 y^2 u / (E (e^E -+ 1)) dy on 256 points of [0, 100]."""
    if fermion not in _DJ:
        u = np.linspace(0.0, 100.0, 256)
        gx, gw = np.polynomial.legendre.leggauss(16)
        e = np.linspace(0.0, 100.0, 1025)
        y = (0.5 * (e[1:] + e[:-1])[:, None] + 0.5 * np.diff(e)[:, None] * gx).reshape(-1)
        w = (0.5 * np.diff(e)[:, None] * gw).reshape(-1)
        v = np.zeros(256)
        for q in range(1, 256):
            E = np.sqrt(y * y + u[q] * u[q])
            v[q] = np.sum(w * y * y * u[q] * np.exp(-E) / (E * (1.0 + np.exp(-E) if fermion else -np.expm1(-E))))
        h, n = u[1] - u[0], 256
        A, r = np.zeros((n, n)), np.zeros(n)
        for i in range(1, n - 1):
            A[i, i - 1:i + 2] = 1.0, 4.0, 1.0
            r[i] = 6.0 * (v[i + 1] - 2.0 * v[i] + v[i - 1]) / h ** 2
        A[0, :3] = A[-1, -3:] = 1.0, -2.0, 1.0
        M = np.linalg.solve(A, r)
        c = np.stack([(M[1:] - M[:-1]) / (6 * h), 0.5 * M[:-1],
                      (v[1:] - v[:-1]) / h - h * (2 * M[:-1] + M[1:]) / 6.0, v[:-1]])
        _DJ[fermion] = torch.from_numpy(c).to(DEV)
    return _DJ[fermion]


def _thermal_vp(x, T, complex_):
    bms, gb, gbg, gf, gfg = COUPLINGS
    lam, (kb, kf) = (LAM_CPLX, COEF_CPLX) if complex_ else (LAM_REAL, COEF_REAL)
    h = 100.0 / 255
    xb = torch.sqrt(bms + 0.5 * gb * gb * x * x + (0.25 * gb * gb + 2.0 / 3.0 * gbg * gbg) * T * T) / T
    xf = torch.sqrt(0.5 * gf * gf * x * x + gfg * gfg * T * T / 6.0) / T

    def dj(c, q):
        q = q.clamp(0.0, 100.0 - 1e-12)
        i = (q / h).long().clamp(0, 254)
        d = q - i * h
        return ((c[0][i] * d + c[1][i]) * d + c[2][i]) * d + c[3][i]

    s = kb * dj(_dj_spline(False), xb) * 0.5 * gb * gb * x / (T * T * xb)
    s += kf * dj(_dj_spline(True), xf) * 0.5 * gf * gf * x / (T * T * xf)
    return lam * x ** 3 - MPHI ** 2 * x + T ** 4 / (2 * math.pi ** 2) * s


def _script_vp(fields, complex_):
    lo, hi = _table_bounds(fields, complex_)
    x = torch.from_numpy(np.linspace(lo, hi, TABLE_SIZE)).to(DEV)
    t = _thermal_vp(x, T_PHYS, complex_)
    dinv = 1.0 / ((hi - lo) / (TABLE_SIZE - 1))
    return lambda q: _lerp(t, lo, dinv, q)


def _polar(vp, eps4=0.0, zn=(0.0, 0.0)):
    """dV/dphi_a of V(|Phi|), eps Re Phi^4 and the Z_N term."""
    def f(a, b):
        rho = torch.sqrt(a * a + b * b)
        safe = rho.clamp(min=1e-30)
        v = vp(rho) / safe
        u, w = v * a, v * b
        if zn[0]:
            t = zn[0] * zn[1] * torch.sin(zn[0] * torch.atan2(b, a)) / (safe * safe)
            on = rho > 1e-20
            u = u - torch.where(on, t * b, 0.0)
            w = w + torch.where(on, t * a, 0.0)
        if eps4:
            u = u + 4 * eps4 * (a ** 3 - 3 * a * b * b)
            w = w + 4 * eps4 * (3 * a * a * b - b ** 3)
        return [u, w]
    return f


def _midpoint(f, force, h1, h2, eta, mu, kick):
    """(phi.., pi..) advanced by h2 with the forces at the midpoint h1."""
    m = len(f) // 2
    i2 = 1.0 / (mu * mu)
    d = force(*f[:m])
    mid = [f[a] + h1 * f[m + a] for a in range(m)]
    vm = [f[m + a] + h1 * (_lap(f[a]) - eta * f[m + a] - d[a] * i2) for a in range(m)]
    d = force(*mid)
    phi = [f[a] + h2 * vm[a] for a in range(m)]
    pi = [f[m + a] + (h2 * (_lap(mid[a]) - eta * vm[a] - d[a] * i2) + kick[a]) for a in range(m)]
    return phi + pi


def _planes(x, storage):
    """A float64 result laid out as the storage."""
    if storage != "f32c":
        return x
    hi = x.float()
    return torch.stack([hi.double(), x - hi.double()])


def exact(case, seed):
    k, st, n = case["kind"], case.get("storage"), int(seed) + 3
    if k == "label":
        return None                                   # whole numbers
    if k in ("step", "cstep"):
        c = k == "cstep"
        f = [_value(x) for x in _toy_state(case, seed, c)]
        vp = _toy_vp(case.get("table") == "2d")
        z = _normals(_shape(case), n, PASS2, int(seed), both=c)
        kick = [_toy_ns() * q for q in (z if c else (z,))]
        force = _polar(vp, EPS4) if c else (lambda a: [vp(a)])
        f = _midpoint(f, force, 0.5 * DT, DT, ETA, 1.0, kick)
        return [_planes(x, st) for x in f]
    if k in ("script", "cscript"):
        c = k == "cscript"
        g = _script_state(case, seed, c)
        vp, f = _script_vp(g, c), [_value(x) for x in g]
        z = _normals(_shape(case), n, PASS2, 0, both=c)
        kick = [_script_ns(ETA_CPLX if c else ETA_REAL) * q for q in (z if c else (z,))]
        zn = (4.0, 1e10) if case.get("zn") else (0.0, 0.0)
        force = _polar(vp, zn=zn) if c else (lambda a: [vp(a)])
        f = _midpoint(f, force, 0.5 * DT_SCRIPT, DT_SCRIPT, ETA_CPLX if c else ETA_REAL, MPHI, kick)
        v = torch.sqrt(f[0] ** 2 + f[1] ** 2) if c else f[0]
        return [_planes(x, st) for x in f] + kick + [float(v.min()), float(v.max()), 0.0]
    if k == "thermal":
        f = [_value(x) for x in _script_state(case, seed, False)]
        h = 0.5 * DT_SCRIPT
        for T, mul in ((T_PHYS, PASS2), (T_PHYS * (1 - 1e-6), PASS4)):
            kick = 0.5 * _script_ns(ETA_REAL) * _normals(_shape(case), n, mul, 0)
            f = _midpoint(f, lambda a: [_thermal_vp(a, T, False)], h, h, ETA_REAL, MPHI, [kick])
        return [_planes(x, st) for x in f]
    if k == "driver":
        return _exact_driver(case, seed)
    if k == "integrator":
        return _exact_integrator(case, seed)
    if k == "winding":
        g = _gen(seed)
        a, b = (_value(_as(_smooth(_shape(case), g, 3), st)) for _ in range(2))
        th = torch.atan2(b, a)

        def wrap(d):
            return (d > math.pi).double() - (d < -math.pi).double()
        e = [wrap(th.roll(-1, d) - th) for d in range(3)]
        w = torch.zeros_like(th)
        for p, q in ((0, 1), (0, 2), (1, 2)):
            w -= e[p] + e[q].roll(-1, p) - e[p].roll(-1, q) - e[q]
        return w
    if k == "ensemble":
        return _exact_ensemble(case, seed)
    return _exact_train(case, seed)


def _exact_driver(case, seed):
    g, sh = _gen(seed), _shape(case)
    f = [_value(_as(x, case["storage"])) for x in (_randn(sh, g, 0.5, 0.4), _randn(sh, g, 1.0))]
    obs = []
    t2, dinv = _toy_table(True)
    for n in range(case["steps"]):
        T = 1.0 - 0.02 * n / 4000
        ns = _toy_ns(T)
        ft = (T - T_LO) * (1.0 / ((T_HI - T_LO) / (NT_TAB - 1)))
        i = min(max(int(ft), 0), NT_TAB - 2)
        row = t2[i] + (ft - i) * (t2[i + 1] - t2[i])
        kick = [ns * _normals(sh, n, PASS2, int(seed))]
        f = _midpoint(f, lambda a: [_lerp(row, LO, dinv, a)], 0.5 * DT, DT, ETA, 1.0, kick)
        p, v = f
        grad = sum(((p.roll(-1, d) - p) ** 2).sum() for d in range(3))
        m, N = (p * p).mean(), p.numel()
        q = (v * v).mean()
        obs.append([float(x) for x in (0.5 * q, 0.5 * grad / N, 0.0, p.mean(), m, q,
                                       (p > 1.0).double().mean(), p.min(), p.max(), 0.0)])
    return [np.array(obs)] + [_planes(x, case["storage"]) for x in f]


def _exact_integrator(case, seed):
    c = case["field"] == "complex"
    g = _script_state(case, seed, c)
    vp = _script_vp(g, c)
    f = [_value(x) for x in g]
    m = 2 if c else 1
    z = _normals(_shape(case), int(seed) + 3, PASS2, 0, both=c)
    z = list(z) if c else [z]
    eta, ns, h = _integrator_eta(case), _integrator_ns(case), 0.5 * DT_SCRIPT
    grad = _polar(vp) if c else (lambda a: [vp(a)])

    def F(p):
        d = grad(*p)
        return [_lap(p[a]) - d[a] / MPHI ** 2 for a in range(m)]
    phi, pi = f[:m], f[m:]
    if case["method"] == "overdamped":
        k = F(phi)
        return [_planes(phi[a] + DT_SCRIPT / eta * k[a] + ns * z[a], case["storage"]) for a in range(m)]
    c1 = math.exp(-eta * DT_SCRIPT)
    c2 = math.sqrt(1.0 - c1 * c1) * ns
    k = F(phi)
    pi = [pi[a] + h * k[a] for a in range(m)]
    phi = [phi[a] + h * pi[a] for a in range(m)]
    pi = [c1 * pi[a] + c2 * z[a] for a in range(m)]
    phi = [phi[a] + h * pi[a] for a in range(m)]
    k = F(phi)
    pi = [pi[a] + h * k[a] for a in range(m)]
    return [_planes(x, case["storage"]) for x in phi + pi]


def _exact_ensemble(case, seed):
    phis, pis, frac = [], [], []
    for (nx, ny, nz), T, E, own in _specs(case, seed):
        sh = (1, nx, ny) if nz == 1 else (nx, ny, nz)
        n = nx * ny * nz
        g = torch.Generator(device=DEV)
        g.manual_seed((int(seed) * 1000003 + own) & (2 ** 63 - 1))
        p = 0.01 * torch.randn(n, dtype=torch.float64, device=DEV, generator=g)
        p = _value(_as(p.view(sh), "f32c"))
        v = torch.zeros_like(p)
        c1, c2, c3 = 0.2 * (T * T - 1.0), -3.0 * E * T, 0.1
        ns = math.sqrt(2.0 * T * 0.05)
        for t in range(case["steps"]):
            p, v = _midpoint([p, v], lambda x: [((c3 * x + c2) * x + c1) * x], 0.025, 0.05, 1.0, 1.0,
                             [ns * _normals(sh, t, PASS2, own)])
        pad = -n % 4
        phis.append(torch.nn.functional.pad(p.reshape(-1), (0, pad)))
        pis.append(torch.nn.functional.pad(v.reshape(-1), (0, pad)))
        frac.append(float((p > 1.0).double().mean()))
    first = None                                      # whole numbers
    return [first, torch.tensor(frac, dtype=torch.float64, device=DEV),
            _planes(torch.cat(phis), "f32c"), _planes(torch.cat(pis), "f32c")]


def _exact_train(case, seed):
    x, t, w = _train_rows(case, seed)
    p = torch.from_numpy(_mlp_params(w)).to(DEV).double().requires_grad_(True)
    t = torch.from_numpy(t).to(DEV).double()
    h, off = torch.nn.functional.pad(torch.from_numpy(x).to(DEV).double(), (0, 10)), 0
    for li in range(4):
        fi, fo = MLP_DIMS[li], MLP_DIMS[li + 1]
        h = h @ p[off:off + fi * fo].view(fi, fo) + p[off + fi * fo:off + fi * fo + fo]
        off += fi * fo + fo
        if li < 3:
            h = torch.nn.functional.silu(h)
    y0, o = h[:, 0], h[:, 1:17]
    loss = (t[:, 2] * (torch.exp(y0) * t[:, 1] - t[:, 0] * y0)).sum()
    loss = loss + ((t[:, 3] / 16.0)[:, None] * (torch.nn.functional.softplus(o) - t[:, 4:] * o)).sum()
    (g,) = torch.autograd.grad(loss / case["rows"], p)
    # the first Adam step: both moments' bias corrections cancel their decay
    return [g, p.detach() - 2e-3 * g / (g.abs() + 1e-8)]
