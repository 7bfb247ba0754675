"""Workloads of the framework as its users call it, for timing.

Each case is one pass through public entry points: sweeps of a reaction
network (host buffers, device buffers, captured graphs, an uneven batch in one
graph, exact SSA), the two fitness paths, and the surrogate's training step
and screening.  Networks, sizes and rates are those of the
benchmark configurations and the tests (bench.py, tests/, fitsearch.py), with
the simulated time cut where a full-length run would take longer than two
seconds.
"""
import ctypes as C
import math

import numpy as np
import torch

import cutauleaping_b200 as ctl
from cutauleaping_b200 import inputs
from cutauleaping_b200 import surrogate as sg

# Networks by name: species, reactions, generator seed and ranges, and the mean
# SSA steps, leaps and leap-free decisions of one simulation up to the instant
# t_ref; counts at other instants go about with (t / t_ref)^power, most of the
# firings falling early (measured; only work() reads these).  `exact` holds the
# SSA steps and their power in exact simulation.
NETWORKS = {
    "schlogl": dict(S=3, R=4, t_ref=5.0, steps=(5097.0, 557.0, 51.0), power=0.6, exact=(18790.0, 1.27)),
    "net12x20": dict(S=12, R=20, seed=0, kw=dict(x0_range=(20, 2000)), t_ref=2.0, steps=(7226.0, 78.0, 73.0),
                     power=0.5, exact=(8336.0, 0.4)),
    "net32x64": dict(S=32, R=64, seed=3, kw={}, t_ref=10.0, steps=(11052.0, 2381.0, 112.0), power=0.3),
    "fit32x64": dict(S=32, R=64, seed=1, kw={}, t_ref=5.0, steps=(40930.0, 214.0, 410.0), power=0.4),
    "net64x128": dict(S=64, R=128, seed=0, kw={}, t_ref=10.0, steps=(46168.0, 222.0, 462.0), power=0.16),
    "net512x1024": dict(S=512, R=1024, seed=0, kw=dict(c_range=(1e-5, 1e-1), x0_range=(1, 100000)), t_ref=2.0,
                        steps=(64.0, 19143.0, 1.0), power=0.29),
}
HIDDEN = (256, 256, 256, 256)


def listed():
    return [
        # a first look at a model: a few dozen simulations through the host call, where launches and latency count
        dict(name="schlogl_host_64", kind="sweep", net="schlogl", n=64, t_end=1.0, samples=20, entry="host"),
        # the bistable model's ensemble, replayed as one graph (the benchmark's first workload)
        dict(name="schlogl_graph_4096", kind="sweep", net="schlogl", n=4096, t_end=5.0, samples=100, entry="graph"),
        # a parameter sweep of the same model: every simulation has its own rate constants
        dict(name="schlogl_rates_65537", kind="sweep", net="schlogl", n=65537, t_end=5.0, samples=100, entry="device",
             sigma=0.5),
        # exact stochastic simulation of a small network (the command line's force_ssa)
        dict(name="net12x20_ssa_8192", kind="sweep", net="net12x20", n=8192, t_end=2.0, samples=50, entry="device",
             ssa=True),
        # an odd-sized exploratory batch of the benchmark network from host buffers, too small to compile a kernel for
        dict(name="net64x128_host_500", kind="sweep", net="net64x128", n=500, t_end=2.0, samples=40, entry="host"),
        # the benchmark's headline workload: 65,536 simulations, 200 samples
        dict(name="net64x128_graph_65536", kind="sweep", net="net64x128", n=65536, t_end=10.0, samples=200,
             entry="graph"),
        # an uneven batch as one graph: a tiny and a mid-sized network, every simulation with its own rates
        dict(name="uneven_graph_65536", kind="uneven", n=32768, t_end=10.0, samples=200, sigma=0.5),
        # the largest network: leap-dominated, groups of several warps per simulation
        dict(name="net512x1024_1184", kind="sweep", net="net512x1024", n=1184, t_end=2.0, samples=50, entry="device"),
        # fitness mode: per-set sample sums from the sweep, then the fitness (what the command line runs)
        dict(name="fitness_mode_16384", kind="sums", net="fit32x64", threads=32, p_rep=64, sets=256, t_end=5.0,
             samples=50, sigma=0.5),
        # fitness of stored samples, the size of one chunk of the parameter search
        dict(name="fitness_256x512", kind="fitness", threads=1, sets=256, p_rep=512, ns=50, s_out=32, reps=1),
        # one optimiser step of the surrogate at the training batch of the parameter search
        dict(name="train_step_16384", kind="train", S=32, batch=16384),
        # screening: every candidate at every instant through the surrogate, scored against the target
        dict(name="screen_100000x50", kind="screen", S=32, n_cand=100000, ns=50, n_par=8),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["sweep", "sweep", "sweep", "sweep", "uneven", "sums", "fitness", "fitness", "train", "screen",
                       "screen"])
    if kind == "sweep":
        net = rng.choice(["schlogl", "schlogl", "net12x20", "net32x64", "net64x128", "net512x1024"])
        hi, t_hi = {"schlogl": (65537, 5.0), "net12x20": (16384, 2.0), "net32x64": (32768, 10.0),
                    "net64x128": (49152, 10.0), "net512x1024": (1184, 2.0)}[net]
        t_end = t_hi * rng.choice([0.2, 0.4, 0.6, 1.0])
        # exact simulation with the networks' own rates only: a perturbed bistable model can fire millions of times
        ssa = net in ("schlogl", "net12x20") and rng.random() < 0.4
        return dict(kind=kind, net=net, n=_log_int(rng, 64, hi), t_end=t_end, samples=rng.randint(20, 100),
                    entry=rng.choice(["host", "device", "graph"]), ssa=ssa,
                    sigma=0.5 if net in ("schlogl", "net32x64") and not ssa and rng.random() < 0.5 else 0.0)
    if kind == "uneven":
        return dict(kind=kind, n=_log_int(rng, 1000, 32768), t_end=10.0 * rng.choice([0.2, 0.5, 1.0]),
                    samples=rng.randint(20, 200), sigma=0.5)
    if kind == "sums":
        return dict(kind=kind, net="fit32x64", threads=rng.choice([1, 16, 32]), p_rep=_log_int(rng, 8, 128),
                    sets=32 * rng.randint(1, 8), t_end=5.0 * rng.choice([0.2, 0.5, 1.0]), samples=rng.randint(20, 50),
                    sigma=0.5)
    if kind == "fitness":
        return dict(kind=kind, threads=rng.choice([1, 1, 16, 64]), sets=64 * _log_int(rng, 1, 4),
                    p_rep=_log_int(rng, 1, 512), ns=rng.randint(20, 100), s_out=rng.randint(1, 32),
                    reps=rng.choice([1, 1, 3]))
    if kind == "train":
        return dict(kind=kind, S=rng.choice([3, 12, 16, 31, 32, 64]), batch=128 * _log_int(rng, 4, 128))
    return dict(kind=kind, S=rng.randint(3, 48), n_cand=_log_int(rng, 200, 100000), ns=rng.randint(20, 50), n_par=8)


# ---- sweeps --------------------------------------------------------------------

def _network(name, n, t_end, samples, sigma, seed):
    """(Network, uniform rates?) with per-simulation log-normal rate factors when sigma > 0."""
    if name == "schlogl":
        net = inputs.schlogl(n, samples=samples, t_end=t_end)
        if sigma:
            net.c = net.c * np.exp(sigma * np.random.default_rng(seed).standard_normal(net.c.shape))
    else:
        d = NETWORKS[name]
        net = inputs.synthetic(d["S"], d["R"], n, seed=d["seed"], t_end=t_end, samples=samples, perturb_sigma=sigma,
                               perturb_seed=seed, **d["kw"])
        if name == "net12x20":  # reaction 0 is a zero-order inflow, as in the fixtures
            net.left[0] = 0
            net.right[0] = 0
            net.right[0, 0] = 1
            net.c[:, 0] = 1.0
    return net, sigma == 0


def _sweep_part(net, uniform, cfg_seed, flags=0):
    model = ctl.Model.create(net.left, net.right, net.feed, net.tvec, net.cs)
    return dict(model=model, n=net.n, cfg=ctl.run_cfg(seed=cfg_seed, uniform_rates=int(uniform), flags=flags),
                X0=torch.from_numpy(np.ascontiguousarray(net.X0, np.int32)).cuda(),
                c=torch.from_numpy(np.ascontiguousarray(net.c, np.float32)).cuda(),
                out=torch.empty((net.n, model.ns, model.s_out), dtype=torch.int32, device="cuda"),
                info=torch.empty((net.n, 40), dtype=torch.uint8, device="cuda"))


def _ptrs(p):
    return p["X0"].data_ptr(), p["c"].data_ptr(), p["out"].data_ptr(), p["info"].data_ptr()


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _prepare_sweep(case, seed):
    net, uniform = _network(case["net"], case["n"], case["t_end"], case["samples"], case.get("sigma", 0.0), seed)
    flags = ctl.FORCE_SSA if case.get("ssa") else 0
    if case["entry"] == "host":
        model = ctl.Model.create(net.left, net.right, net.feed, net.tvec, net.cs)
        return dict(entry="host", model=model, X0=np.ascontiguousarray(net.X0, np.int32),
                    c=np.ascontiguousarray(net.c, np.float32), cfg=ctl.run_cfg(seed=seed, flags=flags))
    p = _sweep_part(net, uniform, seed, flags)
    p["entry"] = case["entry"]
    if case["entry"] == "graph":
        p["graph"] = p["model"].graph(p["n"], *_ptrs(p), 0, p["cfg"])
    return p


def _run_sweep(s):
    if s["entry"] == "host":
        out, info = s["model"].run(s["X0"], s["c"], s["cfg"])
        return {"samples": out.view(np.int32), "info": info.view(np.uint8)}
    if s["entry"] == "graph":
        s["graph"].launch(_stream())
    else:
        s["model"].run_device(s["n"], *_ptrs(s), _stream(), s["cfg"])
    return {"samples": s["out"], "info": s["info"]}


def _prepare_uneven(case, seed):
    parts = []
    for k, (name, t_end, samples) in enumerate([("schlogl", 5.0 * case["t_end"] / 10.0, 100),
                                                ("net32x64", case["t_end"], case["samples"])]):
        net, uniform = _network(name, case["n"], t_end, samples, case["sigma"], seed + k)
        parts.append(_sweep_part(net, uniform, seed + k))
    graph = ctl.graph_multi([(p["model"], p["n"], *_ptrs(p), p["cfg"]) for p in parts])
    return dict(parts=parts, graph=graph)


def _run_uneven(s):
    s["graph"].launch(_stream())
    return [{"samples": p["out"], "info": p["info"]} for p in s["parts"]]


def _sweep_ops(name, n, t_end, ssa_only=False):
    """32-bit operations of a sweep by the convention of the benchmark (per SSA
    step, leap and hand-off decision), at the network's mean step counts."""
    d = NETWORKS[name]
    S, R = d["S"], d["R"]
    nnz = 2.0 * R
    ssa, leaps, hand = (d["exact"][0], 0.0, 0.0) if ssa_only else d["steps"]
    scale = (t_end / d["t_ref"]) ** (d["exact"][1] if ssa_only else d["power"])
    ops = ssa * (6 * R + 2 * nnz / R + 60) + leaps * (44 * R + 6 * nnz + 8 * S + 60) + hand * (4 * R + 4 * nnz + 8 * S)
    return float(n) * scale * ops


def _sweep_bytes(name, n, samples):
    d = NETWORKS[name]
    return n * (4.0 * d["S"] + 4.0 * d["R"] + 4.0 * samples * d["S"] + 40.0)


# ---- fitness ---------------------------------------------------------------------

def _target(rng, ns, reps, s_out, hi):
    """Target counts [ns][1 experiment][reps][s_out]; about one in 64 is zero."""
    t = rng.integers(1, hi, size=(ns, 1, reps, s_out))
    t[rng.random(t.shape) < 1.0 / 64.0] = 0
    return torch.from_numpy(t.astype(np.int32)).cuda()


def _prepare_fitness(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    rng = np.random.default_rng(seed)
    sets, p_rep, ns, so = case["sets"], case["p_rep"], case["ns"], case["s_out"]
    n = sets * p_rep
    # counts around a level of their own per simulation group, instant and species
    level = torch.exp(torch.rand((1, ns, so), device="cuda", generator=g) * 7.0)
    x = torch.randn((n, ns, so), device="cuda", generator=g)
    samples = (level + x * torch.sqrt(level) * 1.5).clamp_(min=0.0).round_().to(torch.int32)
    del x
    return dict(case=case, samples=samples, target=_target(rng, ns, case["reps"], so, 1100),
                exp=torch.zeros(sets, dtype=torch.uint8, device="cuda"),
                fit=torch.zeros(sets, dtype=torch.float64, device="cuda"))


def _check(st, where):
    if st != ctl.OK:
        raise ctl.CtlError(st, where)


def _run_fitness(s):
    c = s["case"]
    _check(ctl.lib().ctl_fitness_device(
        C.c_void_p(s["samples"].data_ptr()), c["ns"], c["s_out"], C.c_void_p(s["target"].data_ptr()),
        C.c_void_p(s["exp"].data_ptr()), 1, c["reps"], c["threads"], c["sets"] * c["p_rep"] // c["threads"], c["p_rep"],
        C.c_void_p(s["fit"].data_ptr()), C.c_void_p(_stream())), "ctl_fitness_device")
    return s["fit"]


def _exact_fitness(case, seed):
    s = _prepare_fitness(case, seed)
    sets, p_rep, th, ns, so = case["sets"], case["p_rep"], case["threads"], case["ns"], case["s_out"]
    # simulation (b * p_rep + par) * threads + t belongs to set b * threads + t
    mean = torch.stack([x.double().mean(0) for x in
                        s["samples"].view(sets // th, p_rep, th, ns, so)]).view(sets, ns, so)
    tgt = s["target"].double().view(1, ns, case["reps"], so)
    d = (tgt - mean.view(sets, ns, 1, so)).abs()
    d = torch.where(tgt != 0, d / tgt.clamp_min(1.0), d)
    return d.sum(dim=(1, 2, 3)) / (ns * so)


def _prepare_sums(case, seed):
    n = case["sets"] * case["p_rep"]
    net, _ = _network(case["net"], 1, case["t_end"], case["samples"], 0.0, seed)
    rng = np.random.default_rng(seed)
    # one set of rate constants per parameter set, p_rep simulations of each
    c_set = net.c[0] * np.exp(case["sigma"] * rng.standard_normal((case["sets"], net.R)))
    gid = np.arange(n)
    th = case["threads"]
    net.X0 = np.tile(net.X0[0], (n, 1))
    net.c = c_set[gid // (th * case["p_rep"]) * th + gid % th]
    model = ctl.Model.create(net.left, net.right, net.feed, net.tvec, net.cs)
    lib = ctl.lib()
    lib.ctl_run_device_sums.argtypes = [C.c_void_p, C.c_void_p, C.c_uint32, C.c_void_p, C.c_void_p, C.c_uint32,
                                        C.c_uint32, C.c_void_p, C.c_void_p, C.c_void_p]
    lib.ctl_fitness_sums_device.argtypes = [C.c_void_p, C.c_uint32, C.c_uint32, C.c_void_p, C.c_void_p] + \
        [C.c_uint32] * 5 + [C.c_void_p, C.c_void_p]
    return dict(case=case, model=model, n=n, cfg=ctl.run_cfg(seed=seed),
                X0=torch.from_numpy(np.ascontiguousarray(net.X0, np.int32)).cuda(),
                c=torch.from_numpy(np.ascontiguousarray(net.c, np.float32)).cuda(),
                sums=torch.empty((case["sets"], model.ns, model.s_out), dtype=torch.int64, device="cuda"),
                info=torch.empty((n, 40), dtype=torch.uint8, device="cuda"),
                target=_target(rng, model.ns, 1, model.s_out, 5000),
                exp=torch.zeros(case["sets"], dtype=torch.uint8, device="cuda"),
                fit=torch.zeros(case["sets"], dtype=torch.float64, device="cuda"))


def _run_sums(s):
    c, lib, m = s["case"], ctl.lib(), s["model"]
    p = lambda k: C.c_void_p(s[k].data_ptr())  # noqa: E731
    _check(lib.ctl_run_device_sums(m.handle, C.byref(s["cfg"]), s["n"], p("X0"), p("c"), c["threads"], c["p_rep"],
                                   p("sums"), p("info"), C.c_void_p(_stream())), "ctl_run_device_sums")
    _check(lib.ctl_fitness_sums_device(p("sums"), m.ns, m.s_out, p("target"), p("exp"), 1, 1, c["threads"],
                                       s["n"] // c["threads"], c["p_rep"], p("fit"), C.c_void_p(_stream())),
           "ctl_fitness_sums_device")
    return {"sums": s["sums"], "info": s["info"], "fitness": s["fit"]}


# ---- the surrogate -----------------------------------------------------------------

def _out_w(S):
    return max(64, (2 * S + 63) // 64 * 64)


def _weights(S, seed):
    """FP32 weights and biases of a network partly trained: the initialisation's
    scales, with biases away from zero.  Padded inputs and outputs are zero."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    dims = (64, *HIDDEN, _out_w(S))
    W, b = [], []
    for l in range(5):
        fan = 9 if l == 0 else dims[l]
        live = 2 * S if l == 4 else dims[l + 1]
        w = torch.zeros(dims[l + 1], dims[l], device="cuda")
        w[:live, :fan] = torch.randn(live, fan, device="cuda", generator=g) * math.sqrt(1.0 / fan) * (0.3 if l == 4 else 1.0)
        v = torch.zeros(dims[l + 1], device="cuda")
        v[:live] = 0.1 * torch.randn(live, device="cuda", generator=g)
        W.append(w)
        b.append(v)
    return W, b


def _net(S, seed):
    W, b = _weights(S, seed)
    net = sg.MLP(S, seed=0)
    zero = lambda ts: [torch.zeros_like(t) for t in ts]  # noqa: E731
    net.load_state(dict(W=W, b=b, Wb=[w.to(torch.bfloat16) for w in W],
                        WbT=[w.t().contiguous().to(torch.bfloat16) for w in W], m=zero(W), v=zero(W), mb=zero(b),
                        vb=zero(b), step_count=0))
    return net


def _batch(case, seed):
    """Scaled inputs [B][64] BF16 and standardised noisy targets [B][S]."""
    g = torch.Generator(device="cuda").manual_seed(seed + 1)
    B, S = case["batch"], case["S"]
    X = torch.zeros(B, sg.IN_PAD, device="cuda")
    X[:, :9] = torch.rand(B, 9, device="cuda", generator=g) * 2.0 - 1.0
    k = torch.arange(S, device="cuda", dtype=torch.float32)
    mean = torch.sin(X[:, :1] * (1.0 + k / 8.0) + X[:, 1:2]) + 0.5 * X[:, 2:3] * X[:, 8:9]
    return X.to(torch.bfloat16), mean + 0.5 * torch.randn(B, S, device="cuda", generator=g)


def _prepare_train(case, seed):
    X, tgt = _batch(case, seed)
    return dict(net=_net(case["S"], seed), X=X, tgt=tgt)


def _run_train(s):
    net = s["net"]
    y = net.forward(s["X"])
    loss, dW, db = net.backward(y, s["tgt"])
    net.adam(dW, db, lr=1e-3)
    return {"y": y, "loss": loss, "dW": dW, "db": db, "W": net.W, "b": net.b}


def _exact_train(case, seed):
    W, b = _weights(case["S"], seed)
    X, tgt = _batch(case, seed)
    S, n = case["S"], case["batch"]
    Wd = [w.to(torch.bfloat16).double().requires_grad_(True) for w in W]
    bd = [v.double().requires_grad_(True) for v in b]
    h = X.double()
    for l in range(4):
        h = torch.nn.functional.silu(h @ Wd[l].t() + bd[l])
    y = h @ Wd[4].t() + bd[4]
    lv = y[:, S:2 * S].clamp(-12.0, 12.0)
    loss = (0.5 * (lv + (tgt.double() - y[:, :S]) ** 2 * torch.exp(-lv))).sum()
    (loss / (n * S)).backward()
    dW, db = [w.grad for w in Wd], [v.grad for v in bd]
    step = lambda p, d: p.double() - 1e-3 * d / (d.abs() + 1e-8)  # noqa: E731  (Adam's first step)
    return {"y": y.detach(), "loss": loss.detach().view(1), "dW": dW, "db": db,
            "W": [step(w, d) for w, d in zip(W, dW)], "b": [step(v, d) for v, d in zip(b, db)]}


def _screen_inputs(case, seed):
    rng = np.random.default_rng(seed)
    S, ns, n_par = case["S"], case["ns"], case["n_par"]
    lo, hi = np.full(n_par, math.log(1e-3)), np.zeros(n_par)
    sc = sg.Scaling(lo, hi, 5.0, rng.uniform(50, 500, S).astype(np.float32), rng.uniform(5, 50, S).astype(np.float32))
    theta = torch.from_numpy(rng.uniform(lo, hi, size=(case["n_cand"], n_par)).astype(np.float32)).cuda()
    tvec = 5.0 * np.arange(1, ns + 1) / ns
    target = rng.integers(1, 800, size=(ns, S)).astype(np.float32)
    return sc, theta, tvec, target


def _prepare_screen(case, seed):
    sc, theta, tvec, target = _screen_inputs(case, seed)
    return dict(net=_net(case["S"], seed), sc=sc, theta=theta, tvec=tvec, target=target)


def _run_screen(s):
    return sg.screen(s["net"], s["theta"], s["tvec"], s["target"], s["sc"])


def _exact_screen(case, seed):
    W, b = _weights(case["S"], seed)
    Wd, bd = [w.to(torch.bfloat16).double() for w in W], [v.double() for v in b]
    sc, theta, tvec, target = _screen_inputs(case, seed)
    S, ns, n_par = case["S"], case["ns"], case["n_par"]
    f64 = lambda a: torch.as_tensor(np.asarray(a, np.float64), device="cuda")  # noqa: E731
    lo, hi, ym, ys, tgt = f64(sc.log_lo), f64(sc.log_hi), f64(sc.y_mean), f64(sc.y_std), f64(target)
    t = 2.0 * f64(tvec) / 5.0 - 1.0
    fit = []
    for a in range(0, theta.shape[0], 4096):
        x = 2.0 * (theta[a:a + 4096].double() - lo) / (hi - lo) - 1.0
        k = x.shape[0]
        h = torch.cat([x[:, None, :].expand(k, ns, n_par), t[None, :, None].expand(k, ns, 1)], 2).reshape(k * ns, n_par + 1)
        h = torch.nn.functional.silu(h @ Wd[0][:, :n_par + 1].t() + bd[0])
        for l in range(1, 4):
            h = torch.nn.functional.silu(h @ Wd[l].t() + bd[l])
        mean = (h @ Wd[4][:S].t() + bd[4][:S]).view(k, ns, S) * ys + ym
        fit.append(((tgt - mean).abs() / torch.where(tgt != 0, tgt, torch.ones_like(tgt))).sum((1, 2)) / (ns * S))
    return torch.cat(fit)


def _mlp_flops_per_row(S):
    return 2.0 * (64 * 256 + 3 * 256 * 256 + 256 * _out_w(S))


# ---- the entry points -----------------------------------------------------------------

def prepare(case, seed):
    return dict(kind=case["kind"], s={"sweep": _prepare_sweep, "uneven": _prepare_uneven, "sums": _prepare_sums,
                                      "fitness": _prepare_fitness, "train": _prepare_train,
                                      "screen": _prepare_screen}[case["kind"]](case, seed))


def run(state):
    return {"sweep": _run_sweep, "uneven": _run_uneven, "sums": _run_sums, "fitness": _run_fitness,
            "train": _run_train, "screen": _run_screen}[state["kind"]](state["s"])


def work(case):
    k = case["kind"]
    if k == "sweep":
        return {"bytes": _sweep_bytes(case["net"], case["n"], case["samples"]),
                "flops": _sweep_ops(case["net"], case["n"], case["t_end"], bool(case.get("ssa")))}
    if k == "uneven":
        n, t = case["n"], case["t_end"]
        return {"bytes": _sweep_bytes("schlogl", n, 100) + _sweep_bytes("net32x64", n, case["samples"]),
                "flops": _sweep_ops("schlogl", n, t / 2.0) + _sweep_ops("net32x64", n, t)}
    if k == "sums":
        n, d = case["sets"] * case["p_rep"], NETWORKS[case["net"]]
        words = case["samples"] * d["S"]
        return {"bytes": n * (4.0 * d["S"] + 4.0 * d["R"] + 40.0) + case["sets"] * (8.0 * words + 8.0) + 4.0 * words,
                "flops": _sweep_ops(case["net"], n, case["t_end"])}
    if k == "fitness":
        words = case["ns"] * case["s_out"]
        return {"bytes": 4.0 * case["sets"] * case["p_rep"] * words + 4.0 * words * case["reps"] + 9.0 * case["sets"],
                "flops": float(case["sets"] * words * (case["p_rep"] + 4 * case["reps"]))}
    per = _mlp_flops_per_row(case["S"])
    if k == "train":
        params = per / 2.0 + 4 * 256 + _out_w(case["S"])
        B = case["batch"]
        return {"bytes": B * (2.0 * 64 + 4.0 * case["S"] + 4.0 * _out_w(case["S"])) + params * (4.0 * 7 + 2.0 * 4),
                "flops": B * (3.0 * per - 2.0 * 64 * 256)}
    rows = case["n_cand"] * case["ns"]
    return {"bytes": case["n_cand"] * (4.0 * case["n_par"] + 8.0) + 4.0 * case["ns"] * case["S"] + per,
            "flops": rows * per}


def exact(case, seed):
    f = {"fitness": _exact_fitness, "train": _exact_train, "screen": _exact_screen}.get(case["kind"])
    return None if f is None else f(case, seed)
