"""What a user of the engine has it do, as cases that can be timed.

Each case is one call (or one replayed batch) through the package's public entry
points, at sizes taken from this repository's benchmark configurations and tests:
the reference-named host functions (arrays in, arrays out), the device-buffer
interface, the ragged batch, and the surrogate network.

    diagram     bifurcation1D            1-D bifurcation diagram: peaks of every point
    dbscan      bifurcation2DDBSCAN      2-D map of DBSCAN cluster counts
    kde         bifurcation2DKDE         2-D map of KDE mode counts
    basin       bifurcation2DDBSCANIC    2-D map over initial conditions, the 5-D
                                         memristive model (the package's default system)
    lle_line    LLE1D                    largest Lyapunov exponent along a line
    lle_map     LLE2D                    largest Lyapunov exponent, 2-D map
    spectrum    LS2D                     full Lyapunov spectrum, 2-D map
    regime      run_device(LLE_REGIME)   LLE and regime class, device buffers
    surrogate   LLE2D_surrogate          the network-predicted, plainly refined map
    batch       Batch.launch             ragged jobs, one captured graph
    train       Mlp.train                Adam steps of the surrogate network
    predict     Mlp.predict_grid         the network's prediction for a whole grid
"""
from __future__ import annotations

import importlib.util
import math
import sys
from pathlib import Path

import numpy as np
import torch

# Parameter sets of the built-in systems (values[0] = 0.5 is the symmetric CD step).
SYSTEMS = {
    "rossler": dict(values=[0.5, 0.2, 0.2, 5.7], idx=[1, 2], ranges=[0.05, 0.35, 0.05, 0.35], ic=[0.1, 0.1, 0.1]),
    "lorenz": dict(values=[0.5, 10.0, 28.0, 8.0 / 3.0], idx=[1, 2], ranges=[5.0, 20.0, 20.0, 200.0],
                   ic=[0.1, 0.1, 0.1]),
    "chen": dict(values=[0.5, 35.0, 3.0, 28.0], idx=[1, 3], ranges=[30.0, 45.0, 20.0, 30.0], ic=[0.1, 0.1, 0.1]),
    "memristive5": dict(values=[8.0, 35.0, 15.0, 0.01, -1.6676, 0.0676, 0.3682, 0.5], idx=[4, 3],
                        ranges=[-6.0, 6.0, -15.0, 15.0], ic=[0.001, 0.0, 0.0, 0.0, 0.0]),
}
# Least FP64 work of one model step (multiply and add counted apart) in the
# cheapest evaluation known to this repository: Chen and Lorenz at s = 1/2,
# Rossler and the 5-D model as written.
STEP_FLOPS = {"rossler": 17, "lorenz": 14, "chen": 14, "memristive5": 66}
NET_WEIGHTS = 256 * 128 + 256 * 256 + 256 * 256 + 17 * 256
NET_PARAMS = NET_WEIGHTS + 3 * 256 + 17


def _cbf():
    """The package, from the tree in the working folder (its folder name holds a dot)."""
    name = "cbf_b200"
    if name not in sys.modules:
        pkg = Path("cudabifurcation3.0_b200").resolve()
        spec = importlib.util.spec_from_file_location(name, pkg / "__init__.py", submodule_search_locations=[str(pkg)])
        mod = importlib.util.module_from_spec(spec)
        sys.modules[name] = mod
        spec.loader.exec_module(mod)
    return sys.modules[name]


# ---- the cases ---------------------------------------------------------------

def listed():
    return [
        # The smallest request: an exponent along a short line of parameters, as an
        # interactive user sweeps one; far below one wave of threads.
        dict(name="lle-line-rossler-150", kind="lle_line", system="rossler", side=150, h=0.01, NT=0.4, tMax=40.0,
             transient=10.0, s=0.5),
        # The 1-D diagram of the paper-style figure: 1000 points, 150 000 steps each,
        # every peak returned.
        dict(name="diagram-rossler-1000", kind="diagram", system="rossler", side=1000, h=0.01, tMax=500.0,
             transient=1000.0, var=0, pre=1, s=0.5),
        # The 2-D cluster-count map of the benchmark.
        dict(name="dbscan-lorenz-1024", kind="dbscan", system="lorenz", side=1024, h=0.005, tMax=200.0,
             transient=500.0, var=0, pre=1, peaks=10000, eps=1e-3, s=0.5),
        # The 2-D mode-count map of the benchmark, four samples per peak.
        dict(name="kde-lorenz-1024", kind="kde", system="lorenz", side=1024, h=0.005, tMax=200.0, transient=500.0,
             var=0, pre=1, peaks=10000, sampling=4, smooth=0.5, s=0.5),
        # Basins of the default 5-D model over two initial conditions, a ragged side.
        dict(name="basin-memristive-231", kind="basin", system="memristive5", side=231, h=0.005, tMax=150.0,
             transient=100.0, var=4, pre=1, peaks=2000, eps=0.05, s=0.5),
        # The largest exponent map that stays within a second or so, full record.
        dict(name="lle-chen-1024", kind="lle_map", system="chen", side=1024, h=0.002, NT=0.5, tMax=1000.0,
             transient=500.0, s=0.5),
        # Spectrum map, a side that is no multiple of anything.
        dict(name="spectrum-lorenz-517", kind="spectrum", system="lorenz", side=517, h=0.005, NT=0.5, tMax=500.0,
             transient=50.0, s=0.5),
        # Plain LLE + regime class on device buffers, a few waves of points.
        dict(name="regime-chen-600", kind="regime", system="chen", side=600, h=0.002, NT=0.5, tMax=500.0,
             transient=250.0, s=0.5),
        # The refined map: labels, training, prediction, recompute rounds.
        dict(name="surrogate-chen-2048", kind="surrogate", system="chen", side=2048, h=0.002, NT=0.5, tMax=250.0,
             transient=125.0, s=0.5),
        # A ragged mix of small and middling maps replayed as one graph.
        dict(name="batch-24", kind="batch", jobs=24, mix=1, low=64, high=256, s=0.5),
        # The network alone: Adam steps at the refined map's minibatch ...
        dict(name="train-4096", kind="train", rows=65536, batch=4096, steps=200),
        # ... and its prediction over a grid.
        dict(name="predict-chen-4096", kind="predict", system="chen", side=4096),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: a kind, its size over the listed range, its options."""
    kind = rng.choice(["lle_line", "diagram", "diagram", "dbscan", "kde", "basin", "lle_map", "spectrum", "regime",
                       "surrogate", "batch", "train", "predict"])
    s = rng.choice([0.5, 0.5, 0.5, 0.3])
    three = rng.choice(["lorenz", "chen", "rossler"])
    h = {"lorenz": 0.005, "chen": 0.002, "rossler": 0.01, "memristive5": 0.005}
    if kind == "lle_line":
        return dict(kind=kind, system=three, side=_log_int(rng, 40, 1000), h=h[three], NT=0.4,
                    tMax=round(rng.uniform(20.0, 100.0), 1), transient=round(rng.uniform(0.0, 50.0), 1), s=s)
    if kind == "diagram":
        return dict(kind=kind, system=three, side=_log_int(rng, 60, 1500), h=h[three],
                    tMax=round(rng.uniform(50.0, 500.0), 1), transient=round(rng.uniform(20.0, 500.0), 1),
                    var=rng.randrange(3), pre=rng.choice([1, 1, 2, 3]), s=s)
    if kind in ("dbscan", "kde"):
        c = dict(kind=kind, system=three, side=_log_int(rng, 48, 800), h=h[three],
                 tMax=round(rng.uniform(50.0, 200.0), 1), transient=round(rng.uniform(50.0, 400.0), 1),
                 var=rng.randrange(3), pre=rng.choice([1, 1, 2]), peaks=rng.choice([300, 2000, 10000]), s=s)
        if kind == "dbscan":
            c.update(eps=rng.choice([1e-3, 0.02, 0.05]))
        else:
            c.update(sampling=rng.choice([2, 4, 6]), smooth=rng.choice([0.05, 0.3, 0.5, 1.0]))
        return c
    if kind == "basin":
        return dict(kind=kind, system="memristive5", side=_log_int(rng, 32, 256), h=0.005,
                    tMax=round(rng.uniform(40.0, 150.0), 1), transient=round(rng.uniform(20.0, 100.0), 1), var=4,
                    pre=rng.choice([1, 2]), peaks=2000, eps=rng.choice([0.01, 0.05]), s=0.5)
    if kind in ("lle_map", "spectrum", "regime"):
        system = three if kind != "regime" else rng.choice(["lorenz", "chen"])
        top = {"lle_map": 700, "spectrum": 500, "regime": 600}[kind]
        return dict(kind=kind, system=system, side=_log_int(rng, 40, top), h=h[system], NT=0.5,
                    tMax=round(rng.uniform(100.0, 400.0), 1), transient=round(rng.uniform(20.0, 200.0), 1), s=s)
    if kind == "surrogate":
        return dict(kind=kind, system="chen", side=rng.randrange(600, 2049), h=0.002, NT=0.5,
                    tMax=round(rng.uniform(60.0, 250.0), 1), transient=round(rng.uniform(50.0, 125.0), 1), s=0.5)
    if kind == "batch":
        low = _log_int(rng, 16, 96)
        return dict(kind=kind, jobs=rng.randrange(4, 33), mix=rng.randrange(2, 10000), low=low, high=low + 150, s=s)
    if kind == "train":
        return dict(kind=kind, rows=_log_int(rng, 5000, 300000), batch=rng.choice([1000, 2048, 4096]),
                    steps=rng.randrange(20, 200))
    return dict(kind=kind, system=three, side=_log_int(rng, 100, 4096))


# ---- inputs ------------------------------------------------------------------

def _model(case, seed, dims):
    """The model a user would pass: initial conditions and the ends of the swept
    ranges vary a little from seed to seed."""
    rng = np.random.default_rng(seed)
    m = SYSTEMS[case["system"]]
    values = list(m["values"])
    values[7 if case["system"] == "memristive5" else 0] = case.get("s", 0.5)
    ic = [float(v * (1.0 + 0.05 * rng.uniform(-1, 1))) for v in m["ic"]]
    ranges = []
    for a in range(dims):
        lo, hi = m["ranges"][2 * a: 2 * a + 2]
        ranges += [lo + 0.01 * (hi - lo) * rng.uniform(), hi - 0.01 * (hi - lo) * rng.uniform()]
    if case["kind"] == "diagram" and case["system"] == "rossler":
        ranges[1] += 0.05  # up to a = 0.4, past the edge of the attractor
    return dict(values=values, ic=ic, ranges=ranges, idx=m["idx"][:dims])


def _batch_specs(case):
    """Ragged jobs: three systems, three tasks, sides, records and steps drawn."""
    rng = np.random.default_rng(case["mix"])
    specs = []
    for _ in range(case["jobs"]):
        system = ["rossler", "lorenz", "chen"][rng.integers(0, 3)]
        task = ["kde", "dbscan", "lle"][rng.integers(0, 3)]
        specs.append(dict(system=system, task=task, side=int(rng.integers(case["low"], case["high"] + 1)),
                          record=float(rng.uniform(40.0, 300.0)), h=float(rng.uniform(0.002, 0.01))))
    return specs


def prepare(case, seed):
    cbf = _cbf()
    kind = case["kind"]
    st = dict(case=case, cbf=cbf)
    if kind == "batch":
        jobs, outs = [], []
        for k, sp in enumerate(_batch_specs(case)):
            m = _model(dict(case, system=sp["system"]), seed + k, 2)
            kw = dict(system=sp["system"], nPts=sp["side"], ranges=m["ranges"], idxMut=m["idx"], ic=m["ic"],
                      values=m["values"], h=sp["h"], tMax=sp["record"], transientTime=50.0, maxValue=1e4)
            if sp["task"] == "lle":
                kw.update(task=cbf.TASK_LLE, NT=0.5, lleEps=1e-8)
            elif sp["task"] == "kde":
                kw.update(task=cbf.TASK_KDE, maxAmountOfPeaks=1000, kdeSampling=4, kdeI1=-60.0, kdeI2=60.0, kdeH=0.5)
            else:
                kw.update(task=cbf.TASK_DBSCAN, maxAmountOfPeaks=1000, dbscanEps=0.05)
            jobs.append(cbf.make_job(**kw))
            outs.append(torch.zeros(sp["side"] ** 2, dtype=torch.float64 if sp["task"] == "lle" else torch.int32,
                                    device="cuda"))
        st.update(outs=outs, stream=torch.cuda.Stream())
        st["batch"] = cbf.Batch(jobs, [o.data_ptr() for o in outs])
        st["batch"].capture(st["stream"].cuda_stream)
        torch.cuda.synchronize()
        return st
    if kind == "train":
        # labelled points of a parameter plane: smooth exponent, classes in bands
        g = torch.Generator(device="cuda").manual_seed(seed)
        n = case["rows"]
        x = torch.rand(n, 4, generator=g, device="cuda") * 2 - 1
        x[:, 0] = 1.0
        x[:, 3] = 0.3
        y = torch.sin(3.0 * x[:, 1]) + 0.5 * torch.cos(7.0 * x[:, 2] + x[:, 1])
        c = torch.clamp(((y + 1.5) * 5.0).to(torch.int32), 0, 15)
        st.update(x=x.contiguous(), y=y.contiguous(), c=c.contiguous(), net=cbf.Mlp(case["batch"], seed=seed % 1000),
                  stream=torch.cuda.Stream())
        torch.cuda.synchronize()
        return st
    if kind == "predict":
        m = _model(case, seed, 2)
        n = case["side"] ** 2
        net = cbf.Mlp(1024, seed=seed % 1000)
        net.set_params(_net_params(seed))
        job = cbf.make_job(task=cbf.TASK_LLE_REGIME, system=case["system"], nPts=case["side"], ranges=m["ranges"],
                           idxMut=m["idx"], ic=m["ic"], values=m["values"], h=0.002, NT=0.5, tMax=10.0,
                           transientTime=10.0, lleEps=1e-8, maxValue=1e4, seedChunk=200000, maxAmountOfPeaks=512,
                           dbscanEps=0.02, regimeTime=5.0, regimeMinAmp=1e-6, regimeChaosLle=0.05,
                           flags=cbf.FLAG_EXACT_GRID)
        st.update(net=net, job=job, stream=torch.cuda.Stream(),
                  lle=torch.empty(n, dtype=torch.float64, device="cuda"),
                  cls=torch.empty(n, dtype=torch.int32, device="cuda"),
                  conf=torch.empty(n, dtype=torch.float32, device="cuda"))
        torch.cuda.synchronize()
        return st
    dims = 1 if kind in ("lle_line", "diagram") else 2
    if kind == "basin":
        m = _model(case, seed, 2)
        rng = np.random.default_rng(seed)
        m["idx"] = [0, 1]
        m["ranges"] = [-0.5 - 0.05 * rng.uniform(), 0.5, -0.5, 0.5 + 0.05 * rng.uniform()]
    else:
        m = _model(case, seed, dims)
    st.update(m, ic=np.array(m["ic"]), values=np.array(m["values"]), ranges=np.array(m["ranges"]),
              idx=np.array(m["idx"], np.int32))
    if kind == "regime":
        n = case["side"] ** 2
        st.update(stream=torch.cuda.Stream(), lle=torch.empty(n, dtype=torch.float64, device="cuda"),
                  cls=torch.empty(n, dtype=torch.int32, device="cuda"))
        st["job"] = cbf.make_job(task=cbf.TASK_LLE_REGIME, system=case["system"], nPts=case["side"],
                                 ranges=m["ranges"], idxMut=m["idx"], ic=m["ic"], values=m["values"], h=case["h"],
                                 NT=case["NT"], tMax=case["tMax"], transientTime=case["transient"], lleEps=1e-8,
                                 maxValue=1e4, seedChunk=200000, maxAmountOfPeaks=512, dbscanEps=0.02,
                                 regimeTime=min(50.0, case["tMax"]), regimeMinAmp=1e-6, regimeChaosLle=0.05)
        torch.cuda.synchronize()
    return st


# ---- one pass ----------------------------------------------------------------

def run(st):
    case, cbf = st["case"], st["cbf"]
    kind = case["kind"]
    if kind == "batch":
        st["batch"].launch(st["stream"].cuda_stream)
        torch.cuda.current_stream().wait_stream(st["stream"])
        return list(st["outs"])
    if kind == "train":
        net = st["net"]
        net.train(st["x"].data_ptr(), st["y"].data_ptr(), st["c"].data_ptr(), case["rows"], case["steps"], 2e-3,
                  horizon=1500, stream=st["stream"].cuda_stream)
        return net.get_params()
    if kind == "predict":
        st["net"].predict_grid(st["job"], 0.8, 1.2, st["lle"].data_ptr(), st["cls"].data_ptr(),
                               st["conf"].data_ptr(), st["stream"].cuda_stream)
        torch.cuda.current_stream().wait_stream(st["stream"])
        return dict(lle=st["lle"], cls=st["cls"], conf=st["conf"])
    if kind == "regime":
        cbf.run_device(st["job"], st["lle"].data_ptr(), st["cls"].data_ptr(), st["stream"].cuda_stream)
        torch.cuda.current_stream().wait_stream(st["stream"])
        return dict(lle=st["lle"], cls=st["cls"])
    ic, ranges, idx, values = st["ic"], st["ranges"], st["idx"], st["values"]
    n, sysname = case["side"], case["system"]
    if kind == "diagram":
        peaks, counts = cbf.bifurcation1D(case["tMax"], n, case["h"], len(ic), ic, ranges, idx, case["var"], 1e4,
                                          case["transient"], values, len(values), case["pre"], system=sysname)
        # the diagram itself: every point's peaks, one after the other, in a plot buffer
        # with room for 256 a point (and more where that does not do)
        total = int(counts.sum())
        room = 256 * n
        while room < total:
            room *= 4
        points = np.zeros(room)
        np.concatenate([p[:c] for p, c in zip(peaks, counts)], out=points[:total])
        return dict(counts=counts, points=points)
    if kind == "dbscan":
        return cbf.bifurcation2DDBSCAN(case["tMax"], n, case["h"], len(ic), ic, ranges, idx, case["var"], 1e4,
                                       case["peaks"], case["transient"], values, len(values), case["pre"],
                                       case["eps"], system=sysname)
    if kind == "basin":
        return cbf.bifurcation2DDBSCANIC(case["tMax"], n, case["h"], len(ic), ic, ranges, idx, case["var"], 1e7,
                                         case["peaks"], case["transient"], values, len(values), case["pre"],
                                         case["eps"], system=sysname)
    if kind == "kde":
        return cbf.bifurcation2DKDE(case["tMax"], n, case["h"], len(ic), ic, ranges, idx, case["var"], 1e4,
                                    case["peaks"], case["transient"], values, len(values), case["pre"],
                                    case["sampling"], -60.0, 60.0, case["smooth"], system=sysname)
    if kind == "surrogate":
        lle, cls, _ = cbf.LLE2D_surrogate(case["tMax"], case["NT"], n, case["h"], 1e-8, ic, len(ic), ranges, idx, 0,
                                          1e4, case["transient"], values, len(values), system=sysname)
        return dict(lle=lle, cls=cls)
    fn = {"lle_line": cbf.LLE1D, "lle_map": cbf.LLE2D, "spectrum": cbf.LS2D}[kind]
    return fn(case["tMax"], case["NT"], n, case["h"], 1e-8, ic, len(ic), ranges, idx, 0, 1e4, case["transient"],
              values, len(values), system=sysname)


# ---- the work a pass cannot do without -----------------------------------------

def _steps(case, kind, record, h, transient, NT=0.5, dim=3):
    skip = int(transient / h)
    if kind in ("lle_line", "lle_map", "regime", "lle"):
        return skip + 2 * int(record / NT) * int(NT / h)
    if kind == "spectrum":
        return skip + (dim + 1) * int(record / NT) * int(NT / h)
    return skip + int(record / h)


def work(case):
    kind = case["kind"]
    if kind == "train":
        b = case["batch"]
        return {"bytes": float(case["rows"] * 24 + 2 * 4 * NET_PARAMS),
                "flops": float(case["steps"]) * b * 2.0 * (3 * NET_WEIGHTS - 256 * 128)}
    if kind == "predict":
        n = case["side"] ** 2
        return {"bytes": float(n * 16 + 4 * NET_PARAMS), "flops": 2.0 * n * NET_WEIGHTS}
    if kind == "batch":
        b = f = 0.0
        for sp in _batch_specs(case):
            n = sp["side"] ** 2
            b += n * (8 if sp["task"] == "lle" else 4)
            f += float(n) * _steps(case, sp["task"], sp["record"], sp["h"], 50.0) * STEP_FLOPS[sp["system"]]
        return {"bytes": b, "flops": f}
    n = case["side"] ** (1 if kind in ("lle_line", "diagram") else 2)
    steps = _steps(case, kind, case["tMax"], case["h"], case["transient"], case.get("NT", 0.5))
    out = {"diagram": 4, "dbscan": 4, "kde": 4, "basin": 4, "spectrum": 24, "regime": 12, "surrogate": 12}.get(kind, 8)
    if kind == "surrogate":
        # a prediction for every point, the plain method for the labels alone
        labels = min(n, 512 * 512 + 65536)
        plain = _steps(case, "lle", case["tMax"], case["h"], case["transient"], case["NT"])
        return {"bytes": float(n * out), "flops": 2.0 * n * NET_WEIGHTS + float(labels) * plain * STEP_FLOPS["chen"]}
    return {"bytes": float(n * out), "flops": float(n) * steps * STEP_FLOPS[case["system"]]}


# ---- values in 64 bits -----------------------------------------------------------

def _net_params(seed):
    """A network with weights of the trained network's scale, flat in the library's
    order: W1 [256 x 128] b1 W2 [256 x 256] b2 W3 [256 x 256] b3 W4 [17 x 256] b4."""
    rng = np.random.default_rng(seed)
    parts = []
    for out, fan in ((256, 128), (256, 256), (256, 256), (17, 256)):
        bound = math.sqrt(6.0 / fan)
        parts += [rng.uniform(-bound, bound, out * fan), rng.uniform(-0.1, 0.1, out)]
    return np.concatenate(parts).astype(np.float32)


def _frequencies():
    """The fixed input frequencies of the network: sums of four bytes of a xorshift
    stream, centred, in sixteenths."""
    mask = (1 << 64) - 1
    state = (0x5EED * 0x9E3779B97F4A7C15 + 1) & mask
    b = np.empty((62, 2))
    for k in range(62):
        for j in range(2):
            state ^= (state << 13) & mask
            state ^= state >> 7
            state ^= (state << 17) & mask
            b[k, j] = (sum((state >> (8 * i)) & 255 for i in range(4)) - 510) / 16.0
    return b


def exact(case, seed):
    """The network's prediction in 64 bits.  The other kinds return counts, or
    follow trajectories for thousands of time units: what those return depends on
    every rounding on the way, so no arithmetic but their own gives their value;
    the trained weights depend on the minibatches the library draws."""
    if case["kind"] != "predict":
        return None
    m = _model(case, seed, 2)
    side = case["side"]
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if dev == "cpu" and side > 512:
        return None
    p = torch.from_numpy(_net_params(seed)).to(dev).double()
    layers, o = [], 0
    for rows, fan in ((256, 128), (256, 256), (256, 256), (17, 256)):
        layers.append((p[o:o + rows * fan].view(rows, fan), p[o + rows * fan:o + rows * fan + rows]))
        o += rows * fan + rows
    freq = torch.from_numpy(_frequencies()).to(dev)
    code = {"rossler": -1.0, "lorenz": 0.0, "chen": 1.0}[case["system"]]
    third = next(i for i in (1, 2, 3) if i not in m["idx"])
    axis = torch.arange(side, device=dev, dtype=torch.float64) * (2.0 / (side - 1)) - 1.0
    lle = torch.empty(side * side, dtype=torch.float64, device=dev)
    conf = torch.empty(side * side, dtype=torch.float64, device=dev)
    chunk = max(1, (1 << 20) // side)
    for r in range(0, side, chunk):
        x2 = axis[r:r + chunk].repeat_interleave(side)
        x1 = axis.repeat(len(x2) // side)
        phase = 2.0 * math.pi * (x1[:, None] * freq[:, 0] + x2[:, None] * freq[:, 1])
        e = torch.empty(len(x1), 128, dtype=torch.float64, device=dev)
        e[:, 0], e[:, 1], e[:, 2], e[:, 3] = code, x1, x2, m["values"][third] / 10.0
        e[:, 4::2], e[:, 5::2] = torch.sin(phase), torch.cos(phase)
        for w, b in layers[:3]:
            z = e @ w.T + b
            e = z * torch.sigmoid(z)
        out = e @ layers[3][0].T + layers[3][1]
        at = slice(r * side, r * side + len(x1))
        lle[at] = out[:, 0] * 1.2 + 0.8
        conf[at] = torch.softmax(out[:, 1:], dim=1).amax(dim=1)
    return dict(lle=lle, cls=None, conf=conf)
