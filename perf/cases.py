"""Performance cases of the PPPM-TDBEM time step: what a program that uses this library calls, over
the sizes it uses it at, through `Solver`, `Batch` and the autograd functions.

Kinds of case (`case["kind"]`):
  static           a body at rest, `steps` time steps in one `Solver.step` call (absorbing boundary or
                   PML, FP32 or the FP64 yardstick).  steps = 1 is the per-step loop of the scene
                   driver, steps = 64 a block of recorded accelerations.  With the PML each block is a
                   clip from rest (the split-field update grows over thousands of steps) and the
                   pressure field is read out after it.
  frame            one 1 kHz motion frame of a moving scene: `update_mesh` and the frame's time
                   steps, then the listener samples.  "plate": a moving sphere over a static
                   plate; "two": two moving spheres.
  batch            scenes of uneven size and length advanced together (`Batch.run`).
  adjoint          forward run and gradient with respect to every acceleration
                   (`autograd.listener_signal`), geometry at rest.
  adjoint_moving   the same through motion frames (`autograd.moving_listener_signal`).
  start            a new scene from its mesh: handle, `set_mesh`, one block of steps, samples; what a
                   program that renders many short clips does per clip.

Every body is a perturbed icosphere with band-limited (100 Hz - 8 kHz) unit-RMS noise accelerations
per vertex averaged to triangles, in a grid sized as the scene driver does; mesh, motion and
accelerations come from the seed.  Eight listeners: seven one to four cells outside the body and one
in the grid's far corner.

`exact` restates the scheme in 64 bits with plain torch tensors (unquantised weights, sums over all
pairs), with the weight caches' refresh criteria, since these decide the signal of a moving scene.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pppm-tdbem_b200", "python"))
from pppm_b200 import Batch, Solver, scenes  # noqa: E402
from pppm_b200.autograd import listener_signal, moving_listener_signal  # noqa: E402

C = 340.3
REFLECT = 0.83
TAPS = 16


def listed():
    return [
        # the scene driver's loop, one time step per call on the smallest benchmark scene: latency
        dict(name="sphere32_step", kind="static", res=32, sub=3, steps=1, pml=0, precision="fp32"),
        # the static benchmark scene, a block of steps per call
        dict(name="sphere32_run", kind="static", res=32, sub=3, steps=64, pml=0, precision="fp32"),
        # an odd grid with a coarse body: nothing divides the tiles
        dict(name="sphere27_run", kind="static", res=27, sub=2, steps=50, pml=0, precision="fp32"),
        # the error yardstick that FP32 results are quoted against
        dict(name="sphere32_fp64_run", kind="static", res=32, sub=3, steps=64, pml=0, precision="fp64"),
        # the split-field PML instead of the absorbing boundary, a clip and its final field
        dict(name="pml48_run", kind="static", res=48, sub=3, steps=64, pml=6, precision="fp32"),
        # a moving scene at an odd resolution, host arrays in as the scene driver has them
        dict(name="moving57_frame", kind="frame", scene="plate", res=57, sub=3, plate=512, host=True, tune=False),
        # the headline benchmark scene, autotuned once after set_mesh as the benchmark does
        dict(name="moving64_frame", kind="frame", scene="plate", res=64, sub=4, plate=1280, host=False, tune=True),
        # the large moving scene: 40960 triangles
        dict(name="large128_frame", kind="frame", scene="two", res=128, sub=5, plate=0, host=False, tune=False),
        # eight scenes of the batch benchmark's ranges, uneven lengths
        dict(name="batch8_run", kind="batch", scenes=8, lo=24, hi=64, steps_lo=40, steps_hi=200),
        # the adjoint benchmark's scene, a shorter run
        dict(name="adjoint48", kind="adjoint", res=48, sub=4, plate=1280, steps=160),
        # a gradient through three motion frames
        dict(name="adjoint_moving64", kind="adjoint_moving", res=64, sub=3, plate=512, frames=3),
        # a short clip of a new scene from its mesh
        dict(name="start48", kind="start", res=48, sub=3, steps=96),
    ]


def draw(rng):
    def logint(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["static", "static", "static", "frame", "frame", "frame", "batch", "adjoint", "adjoint_moving", "start"])
    if kind == "static":
        res = logint(20, 100)
        pml = rng.choice([0, 0, 0, 3, 6])
        prec = rng.choice(["fp32", "fp32", "fp32", "fp64"])
        return dict(kind=kind, res=res, sub=_sub(rng, res), steps=logint(1, 128), pml=pml, precision=prec)
    if kind == "frame":
        if rng.random() < 0.2:
            return dict(kind=kind, scene="two", res=logint(64, 120), sub=4, plate=0, host=rng.random() < 0.5, tune=False)
        res = logint(40, 100)
        return dict(kind=kind, scene="plate", res=res, sub=rng.choice([3, 4]), plate=rng.choice([512, 640, 1280]),
                    host=rng.random() < 0.5, tune=rng.random() < 0.3)
    if kind == "batch":
        lo = logint(20, 32)
        return dict(kind=kind, scenes=rng.randint(2, 8), lo=lo, hi=lo + rng.randint(4, 30), steps_lo=logint(8, 40),
                    steps_hi=logint(48, 200))
    if kind == "adjoint":
        return dict(kind=kind, res=logint(36, 64), sub=rng.choice([3, 4]), plate=rng.choice([512, 1280]), steps=logint(32, 160))
    if kind == "adjoint_moving":
        return dict(kind=kind, res=logint(40, 64), sub=3, plate=rng.choice([512, 640]), frames=rng.randint(2, 3))
    res = logint(24, 64)
    return dict(kind=kind, res=res, sub=rng.choice([2, 3]), steps=logint(16, 128))


def _sub(rng, res):
    """Icosphere subdivision: 320 to 5120 triangles, 20480 where the grid is fine enough that no face
    has more neighbours than the face cache holds."""
    return rng.choice([2, 3, 4] + ([5] if res >= 64 else []))


# ------------------------------------------------------------------------------------ inputs

def _noise(nv, n, dt, gen):
    """Band-limited unit-RMS noise, (n, nv) float32 on the GPU."""
    x = torch.randn((n, nv), generator=gen, device="cuda")
    spec = torch.fft.rfft(x, dim=0)
    f = torch.fft.rfftfreq(n, float(dt), device="cuda")
    spec[(f < 100.0) | (f > 8000.0)] = 0
    y = torch.fft.irfft(spec, n=n, dim=0)
    return y / y.square().mean(0, keepdim=True).sqrt().clamp_min(1e-20)


def _acc(nv, tris, n, dt, seed, silent_from=None):
    """(n, nt) float32 accelerations: vertex noise averaged to triangles; triangles from
    `silent_from` on are silent."""
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    y = _noise(nv, max(n, 512), dt, gen)[:n]
    f = torch.as_tensor(tris, device="cuda", dtype=torch.long)
    a = (y[:, f[:, 0]] + y[:, f[:, 1]] + y[:, f[:, 2]]) / 3
    if silent_from is not None:
        a[:, silent_from:] = 0
    return a.contiguous()


def _target(n, dt, seed):
    """The samples that the gradient cases' loss compares with, (n, 8)."""
    return (1e-2 * _noise(8, max(n, 512), dt, torch.Generator(device="cuda").manual_seed(seed + 1))[:n]).contiguous()


def _listeners(verts, tris, res, h, mn, rng):
    """Seven cells one to four cells outside seven triangles of the first half, and the far corner."""
    v = verts.astype(np.float64)
    out = []
    for k in range(7):
        t = tris[int(rng.integers(0, max(1, len(tris) // 2)))]
        a, b, c = v[t[0]], v[t[1]], v[t[2]]
        n = np.cross(b - a, c - a)
        n /= max(np.linalg.norm(n), 1e-30)
        p = (a + b + c) / 3 + n * float(h) * (1 + k * 0.5)
        out.append(tuple(int(x) for x in np.clip(np.floor((p - mn) / float(h)), 2, res - 3)))
    out.append((int(0.875 * res),) * 3)
    return out


def _sphere(res, sub, seed, pml=0):
    """A perturbed sphere at rest, grid length twice its box (as the static and batch benchmarks)."""
    rng = np.random.default_rng([seed, res, sub])
    v, f = scenes.perturbed_sphere(sub, 0.1, 0.1, rng)
    v = v.astype(np.float32)
    h, mn = scenes.grid_for_bbox(v.min(0), v.max(0), res, 2.0)
    dt = np.float32(0.5 * h / (math.sqrt(3) * C))
    return dict(res=res, h=h, mn=mn, dt=dt, verts=v, tris=f, pml=pml, listeners=_listeners(v, f, res, h, mn, rng))


def _moving(case, seed):
    if case.get("scene", "plate") == "two":
        sc = scenes.LargeScene(res=case["res"], seed=seed, subdivisions=case["sub"])
        silent = None
    else:
        sc = scenes.MovingScene(res=case["res"], seed=seed, subdivisions=case["sub"], plate_tris=case["plate"])
        silent = sc.n_sphere_tris
    v = sc.frame_verts(0)
    rng = np.random.default_rng([seed, 5])
    return sc, silent, _listeners(v, sc.tris, sc.res, sc.h, sc.min_pos, rng)


FRAMES = 12  # motion frames of a frame case's states, walked forth and back


def _solver(inp, stream, precision="fp32"):
    s = Solver(inp["res"], inp["h"], inp["dt"], inp["mn"], pml_width=inp["pml"], precision=precision,
               stream=stream.cuda_stream)
    s.set_mesh(inp["verts"], inp["tris"])
    for c in inp["listeners"]:
        s.add_listener(*c)
    return s


def _batch_inputs(case, seed):
    rng = np.random.default_rng([seed, 77])
    order = np.random.default_rng([case["scenes"], case["lo"], case["hi"], case["steps_lo"], case["steps_hi"]])
    out = []
    for i in range(case["scenes"]):  # sizes and lengths go by the case, shapes by the seed
        res, sub = int(order.integers(case["lo"], case["hi"] + 1)), int(order.integers(2, 5))
        steps = int(order.integers(case["steps_lo"], max(case["steps_lo"], case["steps_hi"]) + 1))
        inp = _sphere(res, sub, int(rng.integers(1 << 30)))
        inp["steps"] = steps
        inp["acc"] = _acc(len(inp["verts"]), inp["tris"], steps, inp["dt"], int(rng.integers(1 << 30)))
        out.append(inp)
    return out


def _plate_inputs(case, seed):
    """The moving scene's first frame held at rest."""
    sc, silent, lis = _moving(case, seed)
    inp = dict(res=sc.res, h=sc.h, mn=sc.min_pos, dt=sc.dt, verts=sc.frame_verts(0), tris=sc.tris, pml=0, listeners=lis)
    return sc, silent, inp


def _rows(case):
    """Rows of a frame's sample buffer: frames differ by a step, and the time step goes by the bodies'
    motion, which goes by the seed."""
    return case["res"] * 6 // 5


def _frame_starts(sc, n):
    return [a for a, _ in scenes.frame_ranges(sc, n)]


def prepare(case, seed):
    kind = case["kind"]
    stream = torch.cuda.Stream()
    st = dict(kind=kind, stream=stream, n=0)
    if kind in ("static", "start"):
        inp = _sphere(case["res"], case["sub"], seed, case.get("pml", 0))
        blocks = 1 if kind == "start" else 4
        acc = _acc(len(inp["verts"]), inp["tris"], blocks * case["steps"], inp["dt"], seed)
        torch.cuda.synchronize()
        st.update(inp=inp, acc=list(acc.split(case["steps"])), steps=case["steps"])
        if kind == "static":
            st["solver"] = _solver(inp, stream, case["precision"])
            st["out"] = torch.empty((case["steps"], 8), device="cuda",
                                    dtype=torch.float64 if case["precision"] == "fp64" else torch.float32)
    elif kind == "frame":
        sc, silent, inp = _plate_inputs(case, seed)
        starts = _frame_starts(sc, FRAMES + 1)
        steps = [starts[f + 1] - starts[f] for f in range(FRAMES + 1)]
        acc = _acc(len(inp["verts"]), sc.tris, 4 * max(steps), sc.dt, seed, silent)
        out = torch.zeros((_rows(case), 8), device="cuda")
        torch.cuda.synchronize()
        s = _solver(inp, stream)
        if case["tune"]:
            s.autotune()
        verts = [sc.frame_verts(f) for f in range(FRAMES + 1)]
        if case["host"]:
            acc = acc.cpu().numpy()
        else:
            verts = [torch.from_numpy(v).cuda() for v in verts]
        st.update(solver=s, acc=acc, verts=verts, steps=steps, out=out)
    elif kind == "batch":
        inps = _batch_inputs(case, seed)
        torch.cuda.synchronize()
        solvers = [_solver(i, stream) for i in inps]
        st.update(solvers=solvers, batch=Batch(solvers), acc=[i["acc"] for i in inps],
                  out=[torch.empty((i["steps"], 8), device="cuda") for i in inps])
    elif kind == "adjoint":
        sc, silent, inp = _plate_inputs(case, seed)
        acc = _acc(len(inp["verts"]), sc.tris, case["steps"], sc.dt, seed, silent)
        target = _target(case["steps"], sc.dt, seed)
        torch.cuda.synchronize()
        st.update(solver=_solver(inp, stream), acc=acc.requires_grad_(True), target=target)
    elif kind == "adjoint_moving":
        sc, silent, inp = _plate_inputs(case, seed)
        starts = _frame_starts(sc, case["frames"])
        n = starts[case["frames"]]
        acc = _acc(len(inp["verts"]), sc.tris, n, sc.dt, seed, silent)
        target = _target(n, sc.dt, seed)
        torch.cuda.synchronize()
        st.update(solver=_solver(inp, stream), acc=acc.requires_grad_(True), target=target,
                  frames=[(starts[f], sc.frame_verts(f)) for f in range(case["frames"])])
    return st


# ------------------------------------------------------------------------------------ one pass

def _frame_of_pass(n):
    """Motion frame of pass n: 1, 2, ..., FRAMES, FRAMES - 1, ..., 0, 1, ..."""
    k = (n + 1) % (2 * FRAMES)
    return k if k <= FRAMES else 2 * FRAMES - k


def run(st):
    with torch.cuda.stream(st["stream"]):
        return _RUN[st["kind"]](st)


def _run_static(st):
    s, a = st["solver"], st["acc"][st["n"] % len(st["acc"])]
    st["n"] += 1
    if st["inp"]["pml"]:
        _restart(s)
        s.step(a)
        return s.series(0, st["steps"], out=st["out"]), s.grid(0)
    s.rewind_listeners()
    s.step(a)
    return s.series(0, st["steps"], out=st["out"])


def _run_frame(st):
    s, n = st["solver"], st["n"]
    f = _frame_of_pass(n)
    k = st["steps"][f]
    a = (n % 4) * max(st["steps"])
    st["n"] += 1
    s.update_mesh(st["verts"][f])
    s.rewind_listeners()
    s.step(st["acc"][a:a + k])
    s.series(0, k, out=st["out"][:k])
    return st["out"]  # rows from k on are the buffer's own


def _run_batch(st):
    for s in st["solvers"]:
        s.rewind_listeners()
    st["batch"].run(st["acc"])
    return [s.series(0, len(o), out=o) for s, o in zip(st["solvers"], st["out"])]


def _restart(s):
    """As a training loop does before each iteration: zero fields, time before the first step."""
    s.reset_fields()
    s.rewind_listeners()
    s.t = -1


def _run_adjoint(st):
    s = st["solver"]
    _restart(s)
    sig, _ = listener_signal(s, st["acc"])
    loss = (sig - st["target"]).square().sum()
    (grad,) = torch.autograd.grad(loss, st["acc"])
    return sig.detach(), grad


def _run_adjoint_moving(st):
    s = st["solver"]
    if st["n"]:
        s.update_mesh(st["frames"][0][1])  # the last iteration's backward left other tables
    st["n"] += 1
    _restart(s)
    sig = moving_listener_signal(s, st["acc"], st["frames"], checkpoint_steps=100)
    loss = (sig - st["target"]).square().sum()
    (grad,) = torch.autograd.grad(loss, st["acc"])
    return sig.detach(), grad


def _run_start(st):
    s = _solver(st["inp"], st["stream"])
    s.step(st["acc"][0])
    out = torch.empty((st["steps"], 8), device="cuda")
    s.series(0, st["steps"], out=out)
    s.close()
    return out


_RUN = dict(static=_run_static, frame=_run_frame, batch=_run_batch, adjoint=_run_adjoint,
            adjoint_moving=_run_adjoint_moving, start=_run_start)


# ------------------------------------------------------------------------------------ work

def _pairs(verts, tris, res, h, mn):
    """(face pairs, (cell, triangle) pairs) of a mesh in its grid."""
    c, _, _, cell, base = _cells(torch.from_numpy(np.asarray(verts, np.float32)), torch.from_numpy(np.asarray(tris)).long(), h, mn)
    cnt = torch.zeros((res + 6,) * 3)
    cnt.index_put_(tuple((cell[:, d] + 3) for d in range(3)), torch.ones(len(cell)), accumulate=True)
    n4 = torch.nn.functional.avg_pool3d(cnt[None, None], 4, 1)[0, 0] * 64  # window starting at the index
    return int(n4[tuple((base[:, d] + 2) for d in range(3))].sum().round()), 27 * len(tris)


def work(case):
    """A time step reads two grid levels and writes one; each triangle's history window, its 54 near-field
    records and each face pair's record (72 B and a 4 B index) enter once per set of tables, since
    nothing in the scheme needs them from memory at every step."""
    kind, b, f = case["kind"], 0.0, 0.0

    def add(inp, steps, updates=0, passes=1, real=4):
        nonlocal b, f
        pf, p3 = _pairs(inp["verts"], inp["tris"], inp["res"], inp["h"], inp["mn"])
        nt, cells = len(inp["tris"]), inp["res"] ** 3
        rec = 76 if real == 4 else 260
        b += passes * (steps * (3 * real * cells + nt * (4 + 2 * real)) + pf * rec + nt * 54 * rec + nt * 32 * real)
        f += passes * steps * (64.0 * (pf + 54 * nt) + 16.0 * cells)
        if inp.get("pml"):
            m, w = inp["res"] - 2, inp["pml"]
            layer = m ** 3 - max(inp["res"] - 2 * w, 0) ** 3
            b += passes * steps * 2 * 6 * real * layer
        if updates:  # new records: nine complex wave numbers, eight points each, both layers
            b += updates * (inp["verts"].size * 4 + nt * 54 * 76)
            f += updates * nt * 27 * 9 * 8 * 40.0

    if kind in ("static", "start"):
        add(_sphere(case["res"], case["sub"], 1, case.get("pml", 0)), case["steps"], updates=kind == "start",
            real=8 if case.get("precision") == "fp64" else 4)
    elif kind == "frame":
        sc, _, inp = _plate_inputs(case, 1)
        add(inp, scenes.frame_ranges(sc, 1)[1][1] - scenes.frame_ranges(sc, 1)[1][0], updates=1)
    elif kind == "batch":
        for inp in _batch_inputs(case, 1):
            add(inp, inp["steps"])
    elif kind == "adjoint":
        _, _, inp = _plate_inputs(case, 1)
        add(inp, case["steps"], passes=2)
        b += 4.0 * case["steps"] * len(inp["tris"])
    else:
        sc, _, inp = _plate_inputs(case, 1)
        n = _frame_starts(sc, case["frames"])[case["frames"]]
        add(inp, n, updates=2 * case["frames"], passes=2)
        b += 4.0 * n * len(inp["tris"])
    return {"bytes": b, "flops": f}


def tolerance(case):
    """The step amplifies rounding from step to step.  Measured with the face-pair and near-field sums in
    another order (one or two steps per pass), over a first and a second pass of every listed case:
    FP32 3e-7 to 6e-6 relative, largest difference 1e-6 to 1.4e-5 of the RMS (the long batch runs
    show the most); FP64 1.5e-15 and 6e-15 over 64 steps, and the FP32 cases' growth (50 roundings)
    gives 1e-14."""
    if case.get("precision") == "fp64":
        return {"rel": 5e-14, "max": 5e-13}
    return {"rel": 2.5e-5, "max": 1e-4}


# ------------------------------------------------------------------------------------ 64-bit restatement

def _cells(v32, f, h, mn):
    """Centres, normals and areas as the step holds them (32 bits), cells and base cells."""
    a, b, c = v32[f[:, 0]], v32[f[:, 1]], v32[f[:, 2]]
    ctr = (a + b + c) / 3
    cr = torch.linalg.cross(b - a, c - a)
    ln = cr.square().sum(1).sqrt()
    m = torch.as_tensor(np.asarray(mn, np.float32), device=v32.device)
    hh = torch.tensor(float(h), dtype=torch.float32, device=v32.device)
    cell = ((ctr - m) / hh).to(torch.long)
    centre = (cell.to(torch.float32) + 0.5) * hh + m
    return ctr, cr / ln[:, None], ln / 2, cell, cell - ((ctr - centre) < 0).long()


class _PairSum(torch.autograd.Function):
    """out[dst] += w . h[src], rows of 32 taps."""

    @staticmethod
    def forward(ctx, h, w, src, dst, n):
        ctx.save_for_backward(w, src, dst)
        ctx.m = h.shape[0]
        out = torch.zeros(n, dtype=h.dtype, device=h.device)
        for i in range(0, len(src), 1 << 21):
            j = slice(i, i + (1 << 21))
            out.index_add_(0, dst[j], (w[j] * h[src[j]]).sum(1))
        return out

    @staticmethod
    def backward(ctx, g):
        w, src, dst = ctx.saved_tensors
        gh = torch.zeros((ctx.m, w.shape[1]), dtype=w.dtype, device=w.device)
        for i in range(0, len(src), 1 << 21):
            j = slice(i, i + (1 << 21))
            gh.index_add_(0, src[j], w[j] * g[dst[j]][:, None])
        return gh, None, None, None, None


class _Exact:
    """The scheme in 64 bits."""

    def __init__(self, inp):
        self.d = "cuda"
        self.res, self.h, self.dt = inp["res"], float(inp["h"]), float(inp["dt"])
        self.mn32 = np.asarray(inp["mn"], np.float32)
        self.mn = torch.as_tensor(self.mn32, device=self.d).double()
        self.h32 = inp["h"]
        self.c, self.reflect = float(np.float32(C)), float(np.float32(REFLECT))
        self.pml = inp["pml"]
        self.f = torch.as_tensor(np.asarray(inp["tris"]), device=self.d).long()
        self.nt = len(self.f)
        dtc = self.dt * self.c
        self.lam = max(dtc ** (3.0 / TAPS), 1e-8 ** (1.0 / (2 * TAPS)))
        s = self.lam * torch.exp(-2j * math.pi * torch.arange(9, device=self.d, dtype=torch.float64) / TAPS)
        self.wave = 0.5 * (s * s - 4 * s + 3) / dtc * 1j
        self.lamn = self.lam ** -torch.arange(TAPS, device=self.d, dtype=torch.float64)
        self.gc = self.pool = None
        n = self.res
        self.p = [torch.zeros(n ** 3, dtype=torch.float64, device=self.d) for _ in range(2)]  # t, t - 1
        self.psi = torch.zeros((n, n, n, 6), dtype=torch.float64, device=self.d)
        self.N = torch.zeros((self.nt, TAPS), dtype=torch.float64, device=self.d)
        self.D = torch.zeros_like(self.N)
        self._boundary()
        cells = [(x * n + y) * n + z for x, y, z in inp["listeners"]]
        self.lis = torch.tensor(cells, device=self.d)

    # ---- weights
    def _layers(self, src, trg, nrm):
        """single and double layer potentials, (..., 9) complex each"""
        d = trg - src
        r2 = d.square().sum(-1)
        zero = r2 == 0
        r = torch.where(zero, torch.ones_like(r2), r2).sqrt()
        ikr = 1j * r[..., None] * self.wave
        e = torch.exp(ikr) / (4 * math.pi * r[..., None])
        dn = -(d * nrm).sum(-1)
        dbl = -e * (1 - ikr) * (dn / (r * r))[..., None]
        keep = (~zero)[..., None]
        return e * keep, dbl * keep

    def _taps(self, spec):
        return torch.fft.irfft(spec, n=TAPS, dim=-1) * self.lamn

    def _tri(self, v):
        a, b, c = v[self.f[:, 0]], v[self.f[:, 1]], v[self.f[:, 2]]
        cr = torch.linalg.cross(b - a, c - a)
        jac = cr.square().sum(1).sqrt()
        return torch.stack([a, b, c], 1), (a + b + c) / 3, cr / jac[:, None], jac

    def _grid_records(self, idx):
        """FDTD-near and BEM-near taps (single, double) of triangles idx: (len, 2, 27, 32)."""
        out = torch.empty((len(idx), 2, 27, 2 * TAPS), dtype=torch.float64, device=self.d)
        off = torch.tensor([[w % 3 - 1, w // 3 % 3 - 1, w // 9 - 1] for w in range(27)], device=self.d)
        nb = torch.tensor([[0, 0, 0], [-1, 0, 0], [1, 0, 0], [0, -1, 0], [0, 1, 0], [0, 0, -1], [0, 0, 1]], device=self.d)
        sc = (self.c * self.dt / self.h) ** 2
        w = torch.tensor([2 - 6 * sc] + [sc] * 6, dtype=torch.float64, device=self.d)
        for i in range(0, len(idx), 1024):
            t = idx[i:i + 1024]
            rel = off[:, None] + nb[None]  # 27, 7, 3
            pts = (self.cell[t][:, None, None] + rel + 0.5) * self.h + self.mn
            s, d = self._layers(self.q[t][:, None, None], pts, self.n[t][:, None, None])
            use = (rel.abs().sum(-1) != 0).double()  # the triangle's own cell has no potential
            half = 0.5 * self.jac[t][:, None, None]
            k = (use * w)[..., None]
            spec = torch.stack([(s * k).sum(2), (d * k).sum(2), s[:, :, 0] * use[:, 0, None], d[:, :, 0] * use[:, 0, None]], 2)
            tp = self._taps(spec * half[..., None])  # (t, 27, 4, 16)
            fd = torch.zeros_like(tp[:, :, :2])
            fd[..., 1:] = tp[:, :, :2, :-1]
            fd[..., 2:] -= tp[:, :, 2:, :-2]
            out[i:i + 1024, 0] = fd.flatten(2)
            out[i:i + 1024, 1] = tp[:, :, 2:].flatten(2)
        return out

    def _singular(self, src, trg, common):
        """Sauter-Schwab panel rules (3 Gauss points per dimension) of face pairs that share `common`
        vertices, vertices as they come."""
        g = torch.tensor([0.774596669241483, 0.0, -0.774596669241483], dtype=torch.float64, device=self.d)
        gw = torch.tensor([0.555555555555554, 0.888888888888889, 0.555555555555554], dtype=torch.float64, device=self.d)
        x, e1, e2, e3 = (t.reshape(-1) for t in torch.meshgrid(*[0.5 * (g + 1)] * 4, indexing="ij"))
        wt = torch.einsum("a,b,c,d->abcd", gw, gw, gw, gw).reshape(-1)
        if common == 3:
            w = x ** 3 * e1 ** 2 * e2
            e12, e123 = e1 * e2, e1 * e2 * e3
            r = [(x, x * (1 - e1 + e12), x * (1 - e123), x * (1 - e1)), (x * (1 - e123), x * (1 - e1), x, x * (1 - e1 + e12)),
                 (x, x * (e1 - e12 + e123), x * (1 - e12), x * (e1 - e12)), (x * (1 - e12), x * (e1 - e12), x, x * (e1 - e12 + e123)),
                 (x * (1 - e123), x * (e1 - e123), x, x * (e1 - e12)), (x, x * (e1 - e12), x * (1 - e123), x * (e1 - e123))]
            f = [w] * 6
        elif common == 2:
            w = x ** 3 * e1 ** 2
            e12, e123 = e1 * e2, e1 * e2 * e3
            r = [(x, x * e1 * e3, x * (1 - e12), x * e1 * (1 - e2)), (x, x * e1, x * (1 - e123), x * e1 * e2 * (1 - e3)),
                 (x * (1 - e12), x * e1 * (1 - e2), x, x * e123), (x * (1 - e123), x * e12 * (1 - e3), x, x * e1),
                 (x * (1 - e123), x * e1 * (1 - e2 * e3), x, x * e12)]
            f = [w] + [w * e2] * 4
        else:
            w = x ** 3 * e2
            r = [(x, x * e1, x * e2, x * e2 * e3), (x * e2, x * e2 * e3, x, x * e1)]
            f = [w] * 2
        out = torch.empty((2, len(src), 9), dtype=torch.complex128, device=self.d)

        def at(tri, u, v):  # (pairs, 3, 3) -> (pairs, nodes, 3)
            return (1 - u)[:, None] * tri[:, None, 0] + (u - v)[:, None] * tri[:, None, 1] + v[:, None] * tri[:, None, 2]

        for i in range(0, len(src), 4096):
            s, t = src[i:i + 4096], trg[i:i + 4096]
            tv, sv, n = self.tri[s], self.tri[t], self.n[s][:, None]
            acc = 0
            for (a, b, c, d), wf in zip(r, f):
                k = (wf * wt)[:, None]
                acc = acc + torch.stack([(z * k).sum(1) for z in self._layers(at(tv, a, b), at(sv, c, d), n)])
            out[:, i:i + 4096] = acc * (self.jac[s] * self.jac[t] / 16)[:, None]
        return out

    def _face_records(self, ctr, nbr):
        """Taps (single, double) of face pairs (source nbr onto face ctr): (len, 32)."""
        out = torch.empty((len(ctr), 2 * TAPS), dtype=torch.float64, device=self.d)
        corner = torch.tensor([[k >> 2, k >> 1 & 1, k & 1] for k in range(8)], device=self.d)
        h32, mn32 = torch.tensor(float(self.h32), device=self.d), torch.as_tensor(self.mn32, device=self.d)
        for i in range(0, len(ctr), 1 << 16):
            c, s = ctr[i:i + (1 << 16)], nbr[i:i + (1 << 16)]
            common = (self.f[c][:, :, None] == self.f[s][:, None, :]).sum((1, 2))
            a = torch.stack(self._layers(self.q[s], self.q[c], self.n[s])) * (0.25 * self.jac[s] * self.jac[c])[:, None]
            close = (self.q[s] - self.q[c]).square().sum(1).sqrt() < self.h * 0.1
            a = a * ~((common == 0) & close)[:, None]
            for k in (1, 2, 3):
                at = (common == k).nonzero()[:, 0]
                if len(at):
                    a[:, at] = self._singular(s[at], c[at], k)
            cells = self.base[c][:, None] + corner
            pts32 = (cells.float() + 0.5) * h32 + mn32
            far = ((pts32 - self.ctr[s][:, None]).abs().double() > self.h * 1.5).any(-1)
            pts = (cells + 0.5) * self.h + self.mn
            ls = self._layers(self.q[s][:, None], pts, self.n[s][:, None])
            k = (-self.interp[c] * far * 0.5 * self.jac[s][:, None])[..., None]
            a = a + torch.stack([(z * k).sum(1) for z in ls])
            out[i:i + (1 << 16)] = self._taps(a).transpose(0, 1).flatten(1)
        return out

    def mesh(self, verts):
        """Lists and weights of a (new) position; records whose geometry moved by less than the caches'
        criteria stay as they were."""
        v32 = torch.as_tensor(np.asarray(verts, np.float32), device=self.d)
        n, nt = self.res, self.nt
        self.tri, self.q, self.n, self.jac = self._tri(v32.double())
        self.ctr, nrm, self.area, self.cell, self.base = _cells(v32, self.f, self.h32, self.mn32)
        lin = (self.cell[:, 0] * n + self.cell[:, 1]) * n + self.cell[:, 2]
        # trilinear weights times the face's area
        u = (self.q - ((self.base + 0.5) * self.h + self.mn)) / self.h
        k = torch.arange(8, device=self.d)
        w = [torch.where((k >> (2 - d) & 1).bool(), u[:, d, None], 1 - u[:, d, None]) for d in range(3)]
        self.interp = 0.5 * self.jac[:, None] * w[0] * w[1] * w[2]
        cb = self.base[:, None] + torch.stack([k >> 2, k >> 1 & 1, k & 1], 1)
        self.corner = (cb[..., 0] * n + cb[..., 1]) * n + cb[..., 2]
        # cell pairs: triangle and each cell of its 3^3 block
        off = torch.tensor([[w % 3 - 1, w // 3 % 3 - 1, w // 9 - 1] for w in range(27)], device=self.d)
        cc = self.cell[:, None] + off
        cells = ((cc[..., 0] * n + cc[..., 1]) * n + cc[..., 2]).flatten()
        self.n3, self.near_dst = torch.unique(cells, return_inverse=True)
        self.near_src = torch.arange(nt, device=self.d).repeat_interleave(27)
        snap = torch.cat([self.ctr, nrm, self.area[:, None]], 1)
        if self.gc is None:
            self.gc, self.snap = self._grid_records(torch.arange(nt, device=self.d)), snap
        else:
            o = self.snap
            m = ((o[:, :3] - snap[:, :3]).square().sum(1).sqrt() > 0.01 * self.h) \
                | ((o[:, 3:6] - snap[:, 3:6]).square().sum(1).sqrt() > 0.01) | ((o[:, 6] - snap[:, 6]).abs() > 0.01 * snap[:, 6])
            at = m.nonzero()[:, 0]
            if len(at):
                self.gc[at] = self._grid_records(at)
                self.snap[at] = snap[at]
        # face pairs: every triangle in the 4^3 block of a face's base cell
        order = lin.argsort()
        count = torch.bincount(lin, minlength=n ** 3)
        start = count.cumsum(0) - count
        ctrs, nbrs = [], []
        for dx in range(-1, 3):
            for dy in range(-1, 3):
                for dz in range(-1, 3):
                    b = self.base + torch.tensor([dx, dy, dz], device=self.d)
                    ok = ((b >= 0) & (b < n)).all(1)
                    bl = ((b[:, 0] * n + b[:, 1]) * n + b[:, 2]).clamp(0, n ** 3 - 1)
                    c = torch.where(ok, count[bl], torch.zeros_like(bl))
                    if not int(c.sum()):
                        continue
                    who = torch.arange(nt, device=self.d).repeat_interleave(c)
                    at = torch.arange(len(who), device=self.d) - (c.cumsum(0) - c)[who] + start[bl[who]]
                    ctrs.append(who)
                    nbrs.append(order[at])
        ctr, nbr = torch.cat(ctrs), torch.cat(nbrs)
        key, o = (ctr * nt + nbr).sort()
        self.fc, self.fn = ctr[o], nbr[o]
        ang = (nrm[self.fn] * nrm[self.fc]).sum(1)
        dist = (self.ctr[self.fn] - self.ctr[self.fc]).square().sum(1).sqrt()
        if self.pool is None:
            self.pool = (key, self._face_records(self.fc, self.fn), ang, dist)
        else:
            pk, pw, pa, pd = self.pool
            allk = torch.unique(torch.cat([pk, key]))
            w = torch.zeros((len(allk), 2 * TAPS), dtype=torch.float64, device=self.d)
            a, dd, have = torch.zeros(len(allk), device=self.d), torch.zeros(len(allk), device=self.d), torch.zeros(len(allk), device=self.d, dtype=torch.bool)
            at = torch.searchsorted(allk, pk)
            w[at], a[at], dd[at], have[at] = pw, pa, pd, True
            here = torch.searchsorted(allk, key)
            redo = ~have[here] | ((a[here] - ang).abs() > 0.01) | ((dd[here] - dist).abs() > 0.01 * dist)
            r = redo.nonzero()[:, 0]
            if len(r):
                w[here[r]] = self._face_records(self.fc[r], self.fn[r])
                a[here[r]], dd[here[r]] = ang[r], dist[r]
            self.pool = (allk, w, a, dd)
        pk, pw = self.pool[:2]
        sign = torch.cat([-torch.ones(TAPS), torch.ones(TAPS)]).double().to(self.d)
        self.face_w = pw[torch.searchsorted(pk, key)] * sign
        self.denom = 0.5 * self.area.double() - torch.zeros(nt, dtype=torch.float64, device=self.d).index_add_(0, self.fc, self.face_w[:, TAPS])
        gw = self.gc * sign
        self.fd_w, self.bm_w = gw[:, 0].reshape(-1, 2 * TAPS), gw[:, 1].reshape(-1, 2 * TAPS)

    # ---- grid
    def _boundary(self):
        n = self.res
        g = torch.arange(1, n - 1, device=self.d)
        xyz = torch.stack(torch.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
        j = (xyz == n - 2).long() - (xyz == 1).long()
        at = (j != 0).any(1)
        xyz, j = xyz[at], j[at]
        st = torch.tensor([n * n, n, 1], device=self.d)
        self.bc, self.bj, self.st = (xyz * st).sum(1), j, st
        on = (j != 0).double()
        coef, c1, c2, c3 = (self.c * self.dt / self.h) ** 2, 1 / self.dt ** 2, self.c / (2 * self.h * self.dt), -self.c ** 2 / (2 * self.h ** 2)
        A = torch.zeros((len(j), 4, 4), dtype=torch.float64, device=self.d)
        A[:, 3, 3] = 1
        A[:, 3, :3] = -coef * on
        for i in range(3):
            A[:, i, 3], A[:, i, i] = c1, c2
            for a in ((i + 1) % 3, (i + 2) % 3):
                A[:, i, a] = c3 * on[:, a]
        self.Ainv = torch.linalg.inv(A)
        self.bk = (coef, c1, c2, c3)

    def _abc(self, cur, prev):
        n = self.res
        c, p = cur.reshape(n, n, n), prev.reshape(n, n, n)
        k = slice(2, n - 2)
        lap = c[1:n - 3, k, k] + c[3:n - 1, k, k] + c[k, 1:n - 3, k] + c[k, 3:n - 1, k] + c[k, k, 1:n - 3] + c[k, k, 3:n - 1] - 6 * c[k, k, k]
        inner = 2 * c[k, k, k] + (self.c * self.dt / self.h) ** 2 * lap - p[k, k, k]
        nxt = torch.nn.functional.pad(inner, (2,) * 6).reshape(-1)
        coef, c1, c2, c3 = self.bk
        b, j = self.bc, self.bj
        pc, pp = cur[b], prev[b]
        up = [cur[b + self.st[d]] for d in range(3)]
        dn = [cur[b - self.st[d]] for d in range(3)]
        inn = [up[d] * (j[:, d] <= 0) + dn[d] * (j[:, d] >= 0) for d in range(3)]
        rhs = []
        for i in range(3):
            y, z = (i + 1) % 3, (i + 2) % 3
            e = -up[i] * (j[:, i] < 0) - dn[i] * (j[:, i] > 0) - prev[b + self.st[i]] * j[:, i] + prev[b - self.st[i]] * j[:, i]
            rhs.append(-c1 * (pp - 2 * pc) - c2 * e - c3 * (inn[y] + inn[z] - 4 * pc))
        rhs.append(-pp + 2 * pc - 6 * coef * pc + coef * (inn[0] + inn[1] + inn[2]))
        r = torch.einsum("nij,nj->ni", self.Ainv, torch.stack(rhs, 1))
        nxt = nxt.index_put((b,), r[:, 3])
        gi = torch.cat([(b + self.st[d] * j[:, d])[j[:, d] != 0] for d in range(3)])
        gv = torch.cat([r[:, d][j[:, d] != 0] for d in range(3)])
        return nxt, cur.index_put((gi,), gv)

    def _pml_step(self, cur, prev):
        n, w, h, dt, cc = self.res, self.pml, self.h, self.dt, self.c
        c, p = cur.reshape(n, n, n), prev.reshape(n, n, n)
        g = torch.arange(n, device=self.d)
        lay = (g < w) | (g >= n - w)
        damp = (lay[:, None, None] | lay[None, :, None] | lay[None, None, :]).double() * float(np.float32(2.0) / np.float32(self.h32))
        ins = torch.zeros((n,) * 3, dtype=torch.bool, device=self.d)
        ins[1:-1, 1:-1, 1:-1] = True
        rhs = torch.zeros_like(c)
        new = self.psi.clone()
        for d in range(3):
            shape = [1, 1, 1]
            shape[d] = n
            upper = (g > n // 2).reshape(shape)

            def ahead(a):  # value at q + sgn e_d
                return torch.where(upper, torch.roll(a, -1, d), torch.roll(a, 1, d))

            def behind(a):
                return torch.where(upper, torch.roll(a, 1, d), torch.roll(a, -1, d))

            f1, f2 = self.psi[..., d], self.psi[..., 3 + d]
            rhs = rhs + (torch.roll(c, -1, d) - 2 * c + torch.roll(c, 1, d)) / h ** 2
            rhs = rhs + (damp * ahead(f2) - behind(damp * f1)) / h
            grad = (ahead(c) - behind(c)) / (2 * h)
            on = ins & (damp != 0)
            new[..., d] = torch.where(on, f1 + cc * dt * (-0.5 * (behind(damp * f1) + damp * f1) - grad), f1)
            new[..., 3 + d] = torch.where(on, f2 + cc * dt * (-0.5 * (behind(damp) * f2 + damp * ahead(f2)) - grad), f2)
        self.psi = new
        return torch.where(ins, 2 * c - p + (cc * dt) ** 2 * rhs, torch.zeros_like(c)).reshape(-1), cur

    def step(self, acc):
        cur, prev = self.p
        nxt, cur = self._pml_step(cur, prev) if self.pml else self._abc(cur, prev)
        zero = torch.zeros((self.nt, 1), dtype=torch.float64, device=self.d)
        before = torch.cat([zero, self.N[:, :-1], zero, self.D[:, :-1]], 1)  # taps at the new time, its own values unknown
        n3 = len(self.n3)
        far = nxt.index_put((self.n3,), nxt[self.n3] - _PairSum.apply(before, self.fd_w, self.near_src, self.near_dst, n3))
        N = torch.cat([acc.double()[:, None], self.N[:, :-1]], 1)
        H = torch.cat([N, zero, self.D[:, :-1]], 1)
        conv = _PairSum.apply(H, self.face_w, self.fn, self.fc, self.nt)
        d = (self.reflect * (self.interp * far[self.corner]).sum(1) + conv) / self.denom
        self.N, self.D = N, torch.cat([d[:, None], self.D[:, :-1]], 1)
        bem = _PairSum.apply(torch.cat([N, self.D], 1), self.bm_w, self.near_src, self.near_dst, n3)
        p = far.index_put((self.n3,), far[self.n3] + 0.98 * bem)
        self.p = [p, cur]
        return p[self.lis]

    def run(self, acc):
        return torch.stack([self.step(a) for a in acc])


def exact(case, seed):
    """What the first pass on these inputs returns, in 64 bits."""
    kind = case["kind"]
    if kind in ("static", "start"):
        inp = _sphere(case["res"], case["sub"], seed, case.get("pml", 0))
        x = _Exact(inp)
        x.mesh(inp["verts"])
        out = x.run(_acc(len(inp["verts"]), inp["tris"], (1 if kind == "start" else 4) * case["steps"], inp["dt"], seed)[: case["steps"]])
        return (out, x.p[0].reshape((case["res"],) * 3)) if inp["pml"] else out
    if kind == "frame":
        sc, silent, inp = _plate_inputs(case, seed)
        starts = _frame_starts(sc, FRAMES + 1)
        steps = [starts[f + 1] - starts[f] for f in range(FRAMES + 1)]
        acc = _acc(len(inp["verts"]), sc.tris, 4 * max(steps), sc.dt, seed, silent)
        x = _Exact(inp)
        x.mesh(sc.frame_verts(0))
        x.mesh(sc.frame_verts(1))
        out = torch.zeros((_rows(case), 8), dtype=torch.float64, device="cuda")
        out[: steps[1]] = x.run(acc[: steps[1]])
        return out
    if kind == "batch":
        out = []
        for inp in _batch_inputs(case, seed):
            x = _Exact(inp)
            x.mesh(inp["verts"])
            out.append(x.run(inp["acc"]))
        return out
    sc, silent, inp = _plate_inputs(case, seed)
    if kind == "adjoint":
        n, frames = case["steps"], [(0, sc.frame_verts(0))]
    else:
        starts = _frame_starts(sc, case["frames"])
        n, frames = starts[case["frames"]], [(starts[f], sc.frame_verts(f)) for f in range(case["frames"])]
    acc = _acc(len(inp["verts"]), sc.tris, n, sc.dt, seed, silent).double().requires_grad_(True)
    target = _target(n, sc.dt, seed)
    x = _Exact(inp)
    sig = []
    ends = [f[0] for f in frames[1:]] + [n]
    for (a, v), b in zip(frames, ends):
        with torch.no_grad():
            x.mesh(v)
        sig.append(x.run(acc[a:b]))
    sig = torch.cat(sig)
    (grad,) = torch.autograd.grad((sig - target.double()).square().sum(), acc)
    return sig.detach(), grad
