"""What the library is asked to do in use, as timed cases.

Every case is a call, or the few calls, that a program makes through openpv_gb300.capi (the
ctypes binding of the C ABI) on buffers and handles that it holds already.  Kinds:

  solve    a whole LCA solve by the batched solver (reset, run, state), BF16 or FP32 form
  step     one LCA timestep composed from the layer and delivery entry points, as a column does it
  pre      compaction of a layer's activity and the presynaptic delivery of its SparseList
  post     postsynaptic delivery of a dense activity (FP32)
  tc       delivery of a dense activity on the tensor cores (post or pre perspective)
  hebbian  the Hebbian weight gradient of a connection
  grad     dL/dW of an unrolled LCA solve
  lif      one LIF layer update

exact() restates each in float64 with plain torch.
"""
import math

import torch

from openpv_gb300 import capi

INF = float("inf")


# ---- the cases ------------------------------------------------------------------------------
def listed():
    return [
        # The benchmark's workload: 256 colour images coded by a 512-feature dictionary, 400
        # timesteps with the last 50 in BF16x3, two half-batch chains.
        {"name": "solve_bf16_b256", "kind": "solve", "prec": "bf16", "nb": 256, "n": 32, "C": 3, "S": 2, "F": 512,
         "steps": 400, "x3": 50, "chains": 2, "vthresh": 0.15},
        # One image through the BF16 solver: the latency of a single solve.
        {"name": "solve_bf16_b1", "kind": "solve", "prec": "bf16", "nb": 1, "n": 32, "C": 1, "S": 2, "F": 64,
         "steps": 200, "x3": 25, "chains": 1, "vthresh": 0.1},
        # The plain FP32 form on a mid-sized batch of colour images.
        {"name": "solve_fp32_b32", "kind": "solve", "prec": "fp32", "nb": 32, "n": 32, "C": 3, "S": 2, "F": 512,
         "steps": 40, "x3": 0, "chains": 1, "vthresh": 0.15},
        # A timestep of a single-image LCA column, call by call: the smallest layers, where the
        # launches and the latency of each kernel are what is paid for.
        {"name": "step_b1", "kind": "step", "nb": 1, "n": 32, "C": 1, "S": 2, "F": 64, "p": 0.1},
        # The same timestep on a batch of colour images and 512 features.
        {"name": "step_b32", "kind": "step", "nb": 32, "n": 32, "C": 3, "S": 2, "F": 512, "p": 0.05},
        # The delivery microbenchmark: a sparse 256-feature layer into 64 features, 7x7.
        {"name": "pre_micro", "kind": "pre", "geo": "one", "nb": 16, "nx": 128, "ny": 128, "nf": 256, "s": 1,
         "p": 7, "qf": 64, "density": 0.01, "spikes": False},
        # Excitatory spikes of the LIF network into its inhibitory layer (many-to-one, stride 2).
        {"name": "pre_exc_inh", "kind": "pre", "geo": "many", "nb": 8, "nx": 256, "ny": 256, "nf": 32, "s": 2,
         "p": 3, "qf": 8, "density": 0.02, "spikes": True},
        # An image batch into 64 features through an 18x18 TransposeConn dictionary (FP32).
        {"name": "post_transpose", "kind": "post", "geo": "many", "nb": 16, "nx": 64, "ny": 64, "nf": 3, "s": 2,
         "p": 9, "qf": 64},
        # Dense delivery of the microbenchmark's connection on the tensor cores.
        {"name": "tc_micro", "kind": "tc", "persp": "post", "nb": 16, "nx": 128, "ny": 128, "nf": 256, "p": 7,
         "qf": 64},
        # A learning step's weight gradient: sparse V1 activity against the error image.
        {"name": "hebbian_b32", "kind": "hebbian", "geo": "up", "nb": 32, "nx": 16, "ny": 16, "nf": 512, "s": 2,
         "p": 8, "qf": 3, "density": 0.05},
        # Dictionary learning by the gradient of the unrolled solve.
        {"name": "grad_b32", "kind": "grad", "nb": 32, "n": 64, "S": 4, "F": 256, "steps": 100, "every": 10},
        # The LIF network's excitatory layer.
        {"name": "lif_b8", "kind": "lif", "nb": 8, "nx": 256, "ny": 256, "nf": 32, "halo": 2, "method": "a"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _pick_geometry(rng, max_work):
    """A connection of the kinds a params file makes: one-to-one with an odd patch, many-to-one, or
    one-to-many, with odd layer sizes and feature counts among them, of at most max_work dense MACs."""
    while True:
        geo = rng.choice(["one", "many", "up"])
        s = 1 if geo == "one" else rng.choice([2, 4])
        small = {"one": rng.choice([1, 3, 5, 7, 9, 11]), "many": rng.randint(2, 9), "up": s * rng.randint(1, 4)}[geo]
        base_x, base_y = _log(rng, 6, 128), _log(rng, 6, 128)
        nx, ny = (base_x * s, base_y * s) if geo == "many" else (base_x, base_y)
        nf, qf = _log(rng, 1, 256), _log(rng, 1, 512)
        if rng.random() < 0.5:
            qf = max(32, qf // 32 * 32) if geo != "up" else rng.choice([1, 3])
        if rng.random() < 0.3:
            nf = rng.choice([1, 3])
        nb = _log(rng, 1, 64)
        work = nb * nx * ny * nf * small * small * qf
        cells = nb * max(nx * ny * nf, nx * ny * qf * (s * s if geo == "up" else 1))
        if work <= max_work and cells <= 1 << 26 and max(nx, ny) <= 512:
            return {"geo": geo, "nb": nb, "nx": nx, "ny": ny, "nf": nf, "s": s, "p": small, "qf": qf}


def draw(rng):
    kind = rng.choice(["solve", "step", "pre", "pre", "post", "post", "tc", "hebbian", "grad", "lif"])
    if kind == "solve":
        S, C = rng.choice([(2, 1), (2, 3), (4, 1)])
        prec = rng.choice(["bf16", "fp32"])
        v1 = 16
        F = 64 * rng.randint(1, 8)
        nb = _log(rng, 1, 256 if prec == "bf16" else 48)
        steps = _log(rng, 10, 200 if prec == "bf16" else 40)
        return {"kind": kind, "prec": prec, "nb": nb, "n": v1 * S, "C": C, "S": S, "F": F, "steps": steps,
                "x3": rng.choice([0, steps // 8]) if prec == "bf16" and S == 2 else 0, "chains": 2 if nb > 1 and rng.random() < 0.5
                else 1, "vthresh": rng.choice([0.1, 0.15])}
    if kind == "step":
        S, C = rng.choice([(2, 1), (2, 3), (4, 1)])
        return {"kind": kind, "nb": _log(rng, 1, 48), "n": S * rng.randint(8, 20), "C": C, "S": S,
                "F": _log(rng, 24, 512), "p": rng.choice([0.02, 0.05, 0.1])}
    if kind == "pre":
        g = _pick_geometry(rng, 3e11)
        return {"kind": kind, **g, "density": rng.choice([0.01, 0.02, 0.05, 0.2]) if g["nf"] > 3 else
                rng.choice([0.03, 1.0]), "spikes": rng.random() < 0.3}
    if kind == "post":
        return {"kind": kind, **_pick_geometry(rng, 6e10)}
    if kind == "tc":
        return {"kind": kind, "persp": rng.choice(["post", "pre"]), "nb": _log(rng, 1, 16), "nx": _log(rng, 16, 128),
                "ny": _log(rng, 16, 128), "nf": 32 * rng.randint(1, 8), "p": rng.choice([3, 5, 7, 9]),
                "qf": 32 * rng.randint(1, 4)}
    if kind == "hebbian":
        return {"kind": kind, **_pick_geometry(rng, 2e9), "density": rng.choice([0.02, 0.05, 0.2, 1.0])}
    if kind == "grad":
        return {"kind": kind, "nb": _log(rng, 2, 32), "n": 64, "S": 4, "F": 32 * rng.randint(1, 8),
                "steps": _log(rng, 10, 100), "every": rng.choice([5, 10])}
    return {"kind": "lif", "nb": _log(rng, 1, 8), "nx": _log(rng, 16, 256), "ny": _log(rng, 16, 256),
            "nf": _log(rng, 1, 32), "halo": rng.randint(0, 4), "method": rng.choice(["a", "b", "o"])}


# ---- geometry ---------------------------------------------------------------------------------
def _axis_start(r, n_pre, n_post, patch):
    """Restricted post index at which the patch of restricted pre index r starts."""
    if n_pre == n_post:
        return r - (patch - 1) // 2
    if n_pre < n_post:
        t = n_post // n_pre
        return r * t - (patch - t) // 2
    s = n_pre // n_post
    return (r - (s // 2) * (patch - 1)) // s


def _margin(n_pre, n_post, patch):
    if n_pre == n_post:
        return (patch - 1) // 2
    if n_pre > n_post:
        return (patch - 1) * (n_pre // n_post) // 2
    return (patch // (n_post // n_pre)) // 2


def _layers(c):
    """(pre, post restricted sizes, patch): the layer the connection leaves and the one it reaches."""
    s = c["s"]
    qx, qy = {"one": (c["nx"], c["ny"]), "many": (c["nx"] // s, c["ny"] // s), "up": (c["nx"] * s, c["ny"] * s)}[c["geo"]]
    # the margin that the presynaptic and (over the post-perspective patch) the postsynaptic delivery ask for
    back = {"one": c["p"], "many": c["p"] * s, "up": c["p"] // s}[c["geo"]]
    m = max(_margin(c["nx"], qx, c["p"]), _margin(qx, c["nx"], back))
    pre = capi.Loc.make(c["nb"], c["nx"], c["ny"], c["nf"], m)
    return pre, capi.Loc.make(c["nb"], qx, qy, c["qf"], 0), c["p"]


def _kernels(pre, post):
    return max(1, pre.nx // post.nx), max(1, pre.ny // post.ny)


def _inner(loc, ext):
    h = loc.halo
    return ext[:, h.up:h.up + loc.ny, h.lt:h.lt + loc.nx, :]


# ---- inputs -----------------------------------------------------------------------------------
def _images(g, nb, n, C):
    """1/f-spectrum images with random phase, zero mean and unit deviation per image."""
    f = torch.fft.fftfreq(n, device="cuda")
    r = torch.sqrt(f[:, None] ** 2 + f[None, :] ** 2)
    r[0, 0] = 1.0
    amp = 1.0 / r
    amp[0, 0] = 0.0
    ph = 2 * math.pi * torch.rand((nb, C, n, n), device="cuda", generator=g)
    img = torch.fft.ifft2(amp * torch.exp(1j * ph)).real.permute(0, 2, 3, 1)
    mu, sd = img.mean(dim=(1, 2, 3), keepdim=True), img.std(dim=(1, 2, 3), keepdim=True)
    return ((img - mu) / sd).float().contiguous()


def _dictionary(g, F, P, C):
    w = torch.randn((F, P, P, C), device="cuda", generator=g)
    return (w / w.square().sum(dim=(1, 2, 3), keepdim=True).sqrt()).contiguous()


def _sparse(g, loc, density, spikes=False):
    """Extended activity: Bernoulli(density) values uniform in (0, 1], or unit spikes; the halo is zero."""
    a = torch.zeros(loc.ext_shape(), device="cuda")
    on = torch.rand(loc.res_shape(), device="cuda", generator=g) < density
    v = torch.ones_like(on, dtype=torch.float32) if spikes else 1.0 - torch.rand(loc.res_shape(), device="cuda", generator=g)
    _inner(loc, a).copy_(on * v)
    return a


def _compaction(loc):
    nb = loc.nbatch
    return (torch.zeros((nb, loc.num_ext, 2), dtype=torch.int32, device="cuda"),
            torch.zeros(nb, dtype=torch.int64, device="cuda"),
            torch.empty(max(1, capi.lib().pvgpu_compact_scratch_bytes(nb, loc.num_ext)), dtype=torch.uint8, device="cuda"))


def _patch(c):
    return {2: 8, 4: 16}[c["S"]]


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _solve_inputs(c, seed):
    g = _gen(seed)
    return _dictionary(g, c["F"], _patch(c), c["C"]), _images(g, c["nb"], c["n"], c["C"])


def _step_locs(c):
    v = c["n"] // c["S"]
    P = _patch(c)
    v1 = capi.Loc.make(c["nb"], v, v, c["F"], _margin(v, c["n"], P))
    return v1, capi.Loc.make(c["nb"], c["n"], c["n"], c["C"], _margin(c["n"], v, P // c["S"])), P


def _step_inputs(c, seed):
    g = _gen(seed)
    v1, er, P = _step_locs(c)
    w, x = _dictionary(g, c["F"], P, c["C"]), _images(g, c["nb"], c["n"], c["C"])
    z = torch.randn(v1.res_shape(), device="cuda", generator=g) * 0.1  # about p of the neurons over threshold
    vt = 0.1 * math.sqrt(2) * float(torch.erfinv(torch.tensor(1.0 - 2 * c["p"])))
    recon = 0.3 * torch.randn(er.res_shape(), device="cuda", generator=g)
    return v1, er, P, w, x, z, float(torch.tensor(vt)), recon


def _conn_inputs(c, seed):
    g = _gen(seed)
    pre, post, p = _layers(c)
    kx, ky = _kernels(pre, post)
    w = 0.05 * torch.randn((kx * ky * pre.nf, p, p, post.nf), device="cuda", generator=g)
    return g, pre, post, p, w


def _post_weights(g, pre, post, p):
    px = p * max(1, pre.nx // post.nx) // max(1, post.nx // pre.nx)
    ph = max(1, post.nx // pre.nx) * max(1, post.ny // pre.ny)
    return 0.05 * torch.randn((ph * post.nf, px, px, pre.nf), device="cuda", generator=g), px


def _tc_layers(c):
    return _layers({**c, "geo": "one", "s": 1})


def _tc_inputs(c, seed):
    g = _gen(seed)
    pre, post, p = _tc_layers(c)
    a = torch.zeros(pre.ext_shape(), device="cuda")
    _inner(pre, a).copy_(torch.rand(pre.res_shape(), device="cuda", generator=g))
    shape = (post.nf, p, p, pre.nf) if c["persp"] == "post" else (pre.nf, p, p, post.nf)
    return pre, post, p, a, 0.05 * torch.randn(shape, device="cuda", generator=g)


def _post_inputs(c, seed):
    g = _gen(seed)
    pre, post, p = _layers(c)
    w, px = _post_weights(g, pre, post, p)
    a = torch.zeros(pre.ext_shape(), device="cuda")
    _inner(pre, a).copy_(torch.randn(pre.res_shape(), device="cuda", generator=g))
    return pre, post, p, px, a, w


def _hebbian_inputs(c, seed):
    g = _gen(seed)
    pre, post, p = _layers(c)
    a = _sparse(g, pre, c["density"])
    r = torch.randn(post.ext_shape(), device="cuda", generator=g)
    return pre, post, p, a, r


def _grad_inputs(c, seed):
    g = _gen(seed)
    return _dictionary(g, c["F"], 16, 1), _images(g, c["nb"], c["n"], 1)


def _lif_inputs(c, seed):
    g = _gen(seed)
    loc = capi.Loc.make(c["nb"], c["nx"], c["ny"], c["nf"], c["halo"])
    n = loc.nbatch * loc.num_res
    rnd = torch.zeros((n, 4), dtype=torch.int32, device="cuda")
    capi.taus_init(rnd, n, seed % 100000 + 1)
    u = lambda lo, hi: lo + (hi - lo) * torch.rand(n, device="cuda", generator=g)  # noqa: E731
    gs = torch.rand((3, n), device="cuda", generator=g) * torch.tensor([[2.0], [1.0], [0.0]], device="cuda")
    return loc, rnd, u(-70, -56), u(-55, -50), u(0, 1), u(0, 1), u(0, 0.5), gs


def prepare(case, seed):
    c, k = case, case["kind"]
    if k == "solve":
        w, x = _solve_inputs(c, seed)
        v = c["n"] // c["S"]
        s = capi.LcaSolver(c["nb"], (c["n"], c["n"], c["C"]), (v, v, c["F"]), _patch(c), c["vthresh"])
        s.set_weights(w)
        if c["chains"] == 2:
            s.set_schedule(chains=2)
        out = torch.empty((2, c["nb"], v, v, c["F"]), device="cuda")
        return {"c": c, "s": s, "x": x, "v": out[0], "a": out[1],
                "prec": capi.LCA_BF16 if c["prec"] == "bf16" else capi.LCA_FP32}
    if k == "step":
        v1, er, P, w, x, v, vt, recon = _step_inputs(c, seed)
        ent, num, scr = _compaction(v1)
        a1, ae = torch.zeros(v1.ext_shape(), device="cuda"), torch.zeros(er.ext_shape(), device="cuda")
        capi.ann_activity(v1, v, vt, 0.0, INF, vt, 0.0, a1)
        gsyn = torch.zeros((2,) + er.res_shape(), device="cuda")
        gsyn[0].copy_(x)
        gsyn[1].copy_(recon)
        return {"c": c, "v1": v1, "er": er, "w": w, "v": v, "a1": a1, "ae": ae, "gsyn": gsyn, "ent": ent, "num": num,
                "scr": scr, "ge": torch.zeros(er.res_shape(), device="cuda"),
                "g1": torch.zeros(v1.res_shape(), device="cuda"), "vt": vt,
                "dt": torch.ones(c["nb"], dtype=torch.float64, device="cuda"),
                "up": capi.conn_desc(er, v1, P // c["S"], P // c["S"]), "down": capi.conn_desc(v1, er, P, P)}
    if k == "pre":
        g, pre, post, p, w = _conn_inputs(c, seed)
        a = _sparse(g, pre, c["density"], c["spikes"])
        ent, num, scr = _compaction(pre)
        return {"c": c, "pre": pre, "conn": capi.conn_desc(pre, post, p, p), "a": a, "w": w, "ent": ent, "num": num,
                "scr": scr, "gsyn": torch.zeros(post.res_shape(), device="cuda")}
    if k == "post":
        pre, post, p, _, a, w = _post_inputs(c, seed)
        return {"c": c, "conn": capi.conn_desc(pre, post, p, p), "a": a, "w": w,
                "gsyn": torch.zeros(post.res_shape(), device="cuda")}
    if k == "tc":
        pre, post, p, a, w = _tc_inputs(c, seed)
        conn = capi.conn_desc(pre, post, p, p)
        ws = torch.empty(capi.deliver_tc_workspace_bytes(conn), dtype=torch.uint8, device="cuda")
        return {"c": c, "conn": conn, "a": a, "w": w, "ws": ws, "gsyn": torch.zeros(post.res_shape(), device="cuda")}
    if k == "hebbian":
        pre, post, p, a, r = _hebbian_inputs(c, seed)
        kx, ky = _kernels(pre, post)
        return {"c": c, "conn": capi.conn_desc(pre, post, p, p), "a": a, "r": r,
                "dw": torch.zeros((kx * ky * pre.nf, p, p, post.nf), device="cuda")}
    if k == "grad":
        w, x = _grad_inputs(c, seed)
        v = c["n"] // c["S"]
        h = capi.LcaGrad(c["nb"], (c["n"], c["n"], 1), (v, v, c["F"]), 16, 0.1, 0.1, c["steps"],
                         checkpoint_every=c["every"])
        return {"c": c, "h": h, "w": w, "x": x, "dw": torch.empty_like(w),
                "loss": torch.zeros(1, dtype=torch.float64, device="cuda")}
    loc, rnd, V, Vth, GE, GI, GIB, gs = _lif_inputs(c, seed)
    return {"c": c, "loc": loc, "rnd": rnd, "V": V, "Vth": Vth, "GE": GE, "GI": GI, "GIB": GIB, "gs": gs,
            "A": torch.zeros(loc.ext_shape(), device="cuda"), "prm": capi.LifParams.make()}


# ---- one pass -----------------------------------------------------------------------------------
def run(st):
    c = st["c"]
    k = c["kind"]
    if k == "solve":
        s = st["s"]
        s.reset()
        s.run(st["x"], c["steps"], x3_steps=c["x3"], precision=st["prec"])
        s.state(st["v"], st["a"])
        return {"V": st["v"], "A": st["a"]}
    if k == "step":
        v1, er, gsyn, vt = st["v1"], st["er"], st["gsyn"], st["vt"]
        # error layer: input minus reconstruction, identity threshold
        capi.gsyn_accumulate(er.nbatch * er.num_res, [1.0, -1.0], gsyn, st["ge"])
        capi.ann_activity(er, st["ge"], -INF, -INF, INF, 0.0, 0.0, st["ae"])
        # V1: delivery of the error, LCA update, threshold
        st["g1"].zero_()
        capi.deliver_post(st["up"], st["ae"], st["w"], st["g1"])
        capi.lca_update(v1, True, st["dt"], 100.0, st["g1"], st["a1"], st["v"])
        capi.ann_activity(v1, st["v"], vt, 0.0, INF, vt, 0.0, st["a1"])
        # V1's activity back to the error layer as a SparseList
        capi.compact_active(st["a1"], v1.nbatch, v1.num_ext, st["ent"], st["num"], scratch=st["scr"])
        gsyn[1].zero_()
        capi.deliver_pre(st["down"], st["w"], gsyn[1], entries=st["ent"], num_active=st["num"])
        return {"ae": st["ae"], "V": st["v"], "A": st["a1"], "recon": gsyn[1]}
    if k == "pre":
        pre = st["pre"]
        capi.compact_active(st["a"], pre.nbatch, pre.num_ext, st["ent"], st["num"], scratch=st["scr"])
        capi.deliver_pre(st["conn"], st["w"], st["gsyn"], entries=st["ent"], num_active=st["num"])
        return {"gsyn": st["gsyn"], "entries": st["ent"], "num": st["num"]}
    if k == "post":
        capi.deliver_post(st["conn"], st["a"], st["w"], st["gsyn"])
        return st["gsyn"]
    if k == "tc":
        f = capi.deliver_post_tc if c["persp"] == "post" else capi.deliver_pre_tc
        f(st["conn"], st["a"], st["w"], st["gsyn"], st["ws"])
        return st["gsyn"]
    if k == "hebbian":
        capi.hebbian_dw(st["conn"], 1.0, st["a"], st["r"], st["dw"])
        return st["dw"]
    if k == "grad":
        st["h"].run(st["w"], st["x"], st["dw"], st["loss"])
        return {"dW": st["dw"], "loss": st["loss"].float()}  # the loss as a training log keeps it
    capi.lif_update(st["loc"], c["method"], st["prm"], 1.0, st["rnd"], st["V"], st["Vth"], st["GE"], st["GI"],
                    st["GIB"], st["gs"], st["A"])
    return {n: st[n] for n in ("V", "Vth", "GE", "GI", "GIB", "A", "rnd")}


# ---- what a pass cannot do without ---------------------------------------------------------------
def work(case):
    c, k = case, case["kind"]
    if k == "solve":
        v = (c["n"] // c["S"]) ** 2
        K = _patch(c) ** 2 * c["C"]
        steps = c["nb"] * c["steps"]
        # V read and written, activity written and read (2 bytes in the BF16 form), the input and the weights
        elt = 12 if c["prec"] == "bf16" else 16
        return {"bytes": steps * (v * c["F"] * elt + 4 * c["n"] ** 2 * c["C"]) + 4 * c["F"] * K,
                "flops": 4 * steps * v * c["F"] * K}
    if k == "step":
        v1, er, P = _step_locs(c)
        n1, ne = v1.nbatch * v1.num_res, er.nbatch * er.num_res
        K = P * P * c["C"]
        return {"bytes": 4 * (4 * n1 + 3 * ne + c["F"] * K) + 8 * c["p"] * n1, "flops": 2 * n1 * K * (1 + c["p"])}
    if k == "grad":
        M = c["nb"] * (c["n"] // c["S"]) ** 2
        T, F = c["steps"], c["F"]
        # forward, recomputation from the checkpoints, adjoint and the two correlations: 8 GEMMs a step
        return {"bytes": 4 * (2 * F * 256 + c["nb"] * c["n"] ** 2 + 2 * M * F * T), "flops": (8 * T + 3) * 2 * M * F * 256}
    if k == "lif":
        return {"bytes": 88 * c["nb"] * c["nx"] * c["ny"] * c["nf"], "flops": 0}
    if k == "tc":
        pre, post, p = _tc_layers(c)
    else:
        pre, post, p = _layers(c)
    n_pre, n_post = pre.nbatch * pre.num_ext, post.nbatch * post.num_res
    wn = pre.nf * p * p * post.nf * max(1, pre.nx // post.nx) ** 2
    # every presynaptic neuron reaches p x p post positions; those outside the layer are not counted
    macs = pre.nbatch * pre.num_res * p * p * post.nf
    if k == "pre":
        nnz = c["density"] * pre.nbatch * pre.num_res
        return {"bytes": 4 * n_pre + 16 * nnz + 8 * n_post + 4 * wn, "flops": 2 * c["density"] * macs}
    if k == "hebbian":
        return {"bytes": 4 * (n_pre + n_post + wn), "flops": 2 * macs * c["density"]}
    return {"bytes": 4 * (n_pre + 2 * n_post + wn), "flops": 2 * macs}


# ---- the same in float64 ---------------------------------------------------------------------------
def _taps(pre, post, p):
    """Per kernel phase (phy, phx) and patch cell (ky, kx): slices of the extended pre layer and of the
    restricted post layer such that their positions pair up one to one."""
    sx, sy = _kernels(pre, post)
    tx, ty = max(1, post.nx // pre.nx), max(1, post.ny // pre.ny)

    def axis(n_ext, border, n_pre, n_post, s, t, phase, k):
        idx = [i for i in range(n_ext) if (i - border) % s == phase]
        pairs = [(i, _axis_start(i - border, n_pre, n_post, p) + k) for i in idx]
        pairs = [(i, q) for i, q in pairs if 0 <= q < n_post]
        if not pairs:
            return None
        (i0, q0), (i1, q1) = pairs[0], pairs[-1]
        return slice(i0, i1 + 1, s), slice(q0, q1 + 1, t)

    for phy in range(sy):
        for phx in range(sx):
            for ky in range(p):
                ay = axis(pre.ny_ext, pre.halo.up, pre.ny, post.ny, sy, ty, phy, ky)
                for kx in range(p):
                    ax = axis(pre.nx_ext, pre.halo.lt, pre.nx, post.nx, sx, tx, phx, kx)
                    if ax and ay:
                        yield phy * sx + phx, ky, kx, ay, ax


def _exact_pre(pre, post, p, a, w):
    out = torch.zeros(post.res_shape(), dtype=torch.float64, device="cuda")
    w = w.double().view(-1, pre.nf, p, p, post.nf)
    for ph, ky, kx, (iy, qy), (ix, qx) in _taps(pre, post, p):
        out[:, qy, qx, :] += a[:, iy, ix, :].double() @ w[ph, :, ky, kx, :]
    return out


def _exact_post(pre, post, px, a, w):
    """Gather: post position r reads a px x px window of pre, weights [phase][post f][px][px][pre f]."""
    out = torch.zeros(post.res_shape(), dtype=torch.float64, device="cuda")
    t = max(1, post.nx // pre.nx)
    w = w.double().view(t * t, post.nf, px, px, pre.nf)
    for py in range(t):
        for pxx in range(t):
            ys, xs = range(py, post.ny, t), range(pxx, post.nx, t)
            y0, x0 = _axis_start(py, post.ny, pre.ny, px) + pre.halo.up, _axis_start(pxx, post.nx, pre.nx, px) + pre.halo.lt
            s = max(1, pre.nx // post.nx)
            for ky in range(px):
                for kx in range(px):
                    win = a[:, y0 + ky:y0 + ky + s * (len(ys) - 1) + 1:s, x0 + kx:x0 + kx + s * (len(xs) - 1) + 1:s, :]
                    out[:, py::t, pxx::t, :] += win.double() @ w[py * t + pxx, :, ky, kx, :].T
    return out


class _Lca:
    """W^T a and W r of an LCA module in float64 by unfold / fold and matrix products."""

    def __init__(self, w, n, S):
        self.P, self.C, self.n, self.S = w.shape[1], w.shape[3], n, S
        self.w = w.double().permute(0, 3, 1, 2).reshape(w.shape[0], -1)  # [F][C*P*P], unfold's order
        self.kw = dict(kernel_size=self.P, stride=S, padding=(self.P - S) // 2)

    def recon(self, a):  # a [nb][L][F] -> [nb][n][n][C]
        d = (a @ self.w).transpose(1, 2)
        return torch.nn.functional.fold(d, (self.n, self.n), **self.kw).permute(0, 2, 3, 1)

    def drive(self, r):
        return torch.nn.functional.unfold(r.permute(0, 3, 1, 2), **self.kw).transpose(1, 2) @ self.w.T


def _f32(v):
    return float(torch.tensor(v, dtype=torch.float32))


def _soft(v, vt):
    return torch.where(v < vt, torch.zeros_like(v), v - vt)


def exact(case, seed):
    c, k = case, case["kind"]
    if k == "solve":
        w, x = _solve_inputs(c, seed)
        if work(c)["flops"] > 1.5e13:
            return None
        m, vt, e = _Lca(w, c["n"], c["S"]), _f32(c["vthresh"]), _f32(math.exp(-1.0 / 100.0))
        side = c["n"] // c["S"]
        v = torch.zeros((c["nb"], side * side, c["F"]), dtype=torch.float64, device="cuda")
        for _ in range(c["steps"]):
            a = _soft(v, vt)
            v = e * v + (1 - e) * (m.drive(x.double() - m.recon(a)) + a)
        shape = (c["nb"], side, side, c["F"])
        return {"V": v.view(shape), "A": _soft(v, vt).view(shape)}
    if k == "step":
        v1, er, P, w, x, v, vt, recon = _step_inputs(c, seed)
        m, e = _Lca(w, c["n"], c["S"]), _f32(math.exp(-1.0 / 100.0))
        err = x.double() - recon.double()
        v0 = v.double().view(c["nb"], -1, c["F"])
        vn = e * v0 + (1 - e) * (m.drive(err) + _soft(v0, vt))
        a = _soft(vn, vt)
        ae, ax = torch.zeros(er.ext_shape(), dtype=torch.float64, device="cuda"), torch.zeros(
            v1.ext_shape(), dtype=torch.float64, device="cuda")
        _inner(er, ae).copy_(err)
        _inner(v1, ax).copy_(a.view(v1.res_shape()))
        return {"ae": ae, "V": vn.view(v1.res_shape()), "A": ax, "recon": m.recon(a)}
    if k == "pre":
        g, pre, post, p, w = _conn_inputs(c, seed)
        a = _sparse(g, pre, c["density"], c["spikes"])
        return {"gsyn": _exact_pre(pre, post, p, a, w), "entries": None, "num": None}
    if k == "post":
        pre, post, p, px, a, w = _post_inputs(c, seed)
        return _exact_post(pre, post, px, a, w)
    if k == "tc":
        pre, post, p, a, w = _tc_inputs(c, seed)
        return _exact_post(pre, post, p, a, w) if c["persp"] == "post" else _exact_pre(pre, post, p, a, w)
    if k == "hebbian":
        pre, post, p, a, r = _hebbian_inputs(c, seed)
        kx_, ky_ = _kernels(pre, post)
        dw = torch.zeros((kx_ * ky_, pre.nf, p, p, post.nf), dtype=torch.float64, device="cuda")
        r = _inner(post, r)
        for ph, ky, kx, (iy, qy), (ix, qx) in _taps(pre, post, p):
            A, R = a[:, iy, ix, :].double().reshape(-1, pre.nf), r[:, qy, qx, :].double().reshape(-1, post.nf)
            dw[ph, :, ky, kx, :] = A.T @ R
        return dw.view(-1, p, p, post.nf)
    if k == "grad":
        w, x = _grad_inputs(c, seed)
        wd = w.double().requires_grad_(True)
        m, vt, e = _Lca(wd, c["n"], c["S"]), _f32(0.1), _f32(math.exp(-1.0 / 100.0))
        L = (c["n"] // c["S"]) ** 2
        v = torch.zeros((c["nb"], L, c["F"]), dtype=torch.float64, device="cuda")
        for _ in range(c["steps"]):
            a = _soft(v, vt)
            v = e * v + (1 - e) * (m.drive(x.double() - m.recon(a)) + a)
        a = _soft(v, vt)
        loss = 0.5 * (x.double() - m.recon(a)).square().sum() + vt * a.abs().sum()
        loss.backward()
        return {"dW": wd.grad, "loss": loss.detach().reshape(1)}
    return _exact_lif(c, seed)


def _exact_lif(c, seed):
    loc, _, v, vth, ge, gi, gib, gs = (t.double() if isinstance(t, torch.Tensor) and t.is_floating_point() else t
                                       for t in _lif_inputs(c, seed))
    q = capi.LifParams.DEFAULTS
    cap, decay = 10.0, lambda tau: _f32(math.exp(-1.0 / tau))  # noqa: E731

    def v_inf(e, i, b):
        return (q["Vrest"] + q["Vexc"] * e + q["Vinh"] * i + q["VinhB"] * b) / (1 + e + i + b)

    if c["method"] == "o":
        ge, gi, gib = ((s + g * decay(t)).clamp(max=cap) for s, g, t in
                       zip(gs, (ge, gi, gib), (q["tauE"], q["tauI"], q["tauIB"])))
        inf = v_inf(ge, gi, gib)
        v = inf + (v - inf) * torch.exp(-(1.0 / q["tau"]) * (1 + ge + gi + gib))
    else:
        e0, i0, b0 = ge + gs[0], gi + gs[1], gib + gs[2]
        tau0, inf0 = q["tau"] / (1 + e0 + i0 + b0), v_inf(e0, i0, b0)
        e0, i0, b0 = (t.clamp(max=cap) for t in (e0, i0, b0))
        ge, gi, gib = e0 * decay(q["tauE"]), i0 * decay(q["tauI"]), b0 * decay(q["tauIB"])
        if c["method"] == "b":
            d = lambda u, e, i, b: (1 + e + i + b) * (v_inf(e, i, b) - u) / q["tau"]  # noqa: E731
            d1 = d(v, e0, i0, b0)
            v = v + (d1 + d(v + d1, ge, gi, gib)) * 0.5
        else:
            tau1, inf1 = q["tau"] / (1 + ge + gi + b0), v_inf(ge, gi, gib)
            slope, ratio = tau1 - tau0, tau1 / tau0
            f1 = torch.where(slope == 0, torch.exp(-1 / tau0), ratio ** (-1 / slope))
            f2 = torch.where(slope == -1, tau0 * torch.log(ratio + 1), (1 - tau0 * (1 - f1)) / (1 + slope))
            v = f1 * v + f2 * inf0 + (1 - f1 - f2) * inf1
    vth = q["VthRest"] + (vth - q["VthRest"]) * decay(q["tauVth"])
    fired = v > vth
    A = torch.zeros(loc.ext_shape(), dtype=torch.float64, device="cuda")
    _inner(loc, A).copy_(fired.view(loc.res_shape()))
    return {"V": torch.where(fired, torch.full_like(v, q["Vrest"]), v), "Vth": vth + fired * q["deltaVth"], "GE": ge,
            "GI": gi, "GIB": gib + fired * q["deltaGIB"], "A": A, "rnd": None}
