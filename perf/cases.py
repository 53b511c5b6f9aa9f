"""The work that users of the near-field library have it do, as measurable cases.

A case names an entry point, a box (particles per side, cells per side,
uniform or clustered), a softening and the options in use:

  sweep     nf_box_forces: accelerations of a box resident in HBM, into device
            memory (the whole box, or `slabs` x-slabs of it)
  kick      nf_box_kick: the same sweep fused with the far field, the rescale
            and the two half kicks
  step      nf_box_step: pinned host positions in, accelerations out to pinned
            host memory, pipelined over slab chunks
  timestep  nf_box_create + nf_box_forces + nf_box_destroy: one step of a
            simulation whose particles have moved between cells, so that the
            cell table is new; positions already on the device
  driver    the NearFieldDriver mirror over every slab, from host slabs into
            the host AccSlabs (ExecuteSlab, SlabDone, Finalize)
  serve     nf_server: requests for every slab of two resident boxes, in a
            mixed order, results into pinned host memory
  noalloc   nf_forces_noalloc: one small box, no allocation

Boxes are generated on the GPU from the seed: 40 % uniform background and 60 %
in NFW clumps (clustered), or uniform; softening length 1/40 of the mean
spacing; where the density channel is on, its radius is 0.2 of a cell.
"""
import ctypes
import importlib.util
import math
import pathlib
import sys
import time

import numpy as np
import torch

ROOT = pathlib.Path(__file__).resolve().parents[1]
PACKAGE = ROOT / "abacus-public_b200"


def _package():
    """The package directory has a dash in its name: it is loaded by path."""
    if "abacus_public_b200" not in sys.modules:
        spec = importlib.util.spec_from_file_location(
            "abacus_public_b200", PACKAGE / "__init__.py",
            submodule_search_locations=[str(PACKAGE)])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["abacus_public_b200"] = mod
        spec.loader.exec_module(mod)
    from abacus_public_b200 import capi, synth
    return capi, synth


PLUMMER, SINGLE_SPLINE, CUBIC_SPLINE, CUBIC_PLUMMER = range(4)


def _case(name, entry, n_side, cpd, clustered, softening=SINGLE_SPLINE, density=False,
          radius=2, record=4, slabs=0):
    c = dict(entry=entry, n_side=n_side, cpd=cpd, clustered=clustered, softening=softening,
             density=density, radius=radius, record=record, slabs=slabs)
    return dict(name=name, **c) if name else c


def listed():
    return [
        # the smallest call: a few thousand particles inside another framework's memory
        _case("noalloc_16", "noalloc", 16, 7, False, PLUMMER),
        # the CPU-checkable box of the tests and the benchmark: launch and tail count
        _case("sweep_uniform_64", "sweep", 64, 17, False, PLUMMER),
        # the clustered box at an ordinary size, the default softening
        _case("sweep_clustered_128", "sweep", 128, 33, True),
        # the benchmark's clustered 256^3 box: the largest
        _case("sweep_clustered_256", "sweep", 256, 65, True),
        # the cubic spline build of the reference, ragged sizes, three-float records
        _case("sweep_cubic_spline_75", "sweep", 75, 19, False, CUBIC_SPLINE, record=3),
        # the reference's default build: single spline with the density channel
        _case("sweep_density_100", "sweep", 100, 25, True, density=True),
        # near field and kick of a simulation step in one call
        _case("kick_clustered_128", "kick", 128, 33, True),
        # end to end from pinned host memory, same cell counts
        _case("step_uniform_160", "step", 160, 41, False),
        # end to end on the device with new cell counts, as after a drift
        _case("timestep_clustered_96", "timestep", 96, 25, True),
        # the drop-in as abacus runs it: host slabs in, AccSlabs out
        _case("driver_uniform_64", "driver", 64, 17, False, PLUMMER),
        _case("driver_density_clustered_96", "driver", 96, 25, True, density=True),
        # every slab of two resident boxes, requested in a mixed order
        _case("serve_2x45", "serve", 180, 45, True),
    ]


#: particles per side by entry point and kind of box (uniform, clustered)
RANGES = {"noalloc": ((8, 40), (8, 40)), "sweep": ((24, 220), (24, 160)),
          "kick": ((24, 200), (24, 140)), "step": ((32, 200), (32, 140)),
          "timestep": ((24, 160), (24, 110)), "driver": ((24, 110), (24, 100)),
          "serve": ((60, 170), (60, 140))}


def draw(rng):
    entry = rng.choice(["sweep", "sweep", "kick", "step", "timestep", "driver", "driver",
                        "serve", "noalloc"])
    clustered = rng.random() < 0.6
    lo, hi = RANGES[entry][clustered]
    n_side = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    # 20 to 110 particles a cell, an odd number of cells
    cpd = int(round(n_side / rng.uniform(20.0, 110.0) ** (1 / 3)))
    cpd = max(5, cpd | 1)
    cpd = min(cpd, 63 if entry == "driver" else 75)
    softening = rng.choice([PLUMMER, SINGLE_SPLINE, SINGLE_SPLINE, SINGLE_SPLINE, CUBIC_SPLINE,
                            CUBIC_PLUMMER])
    density = rng.random() < 0.25
    record = 4 if density or rng.random() < 0.8 else 3
    radius = 1 if rng.random() < 0.1 and entry != "driver" else 2
    slabs = rng.randint(1, cpd) if entry == "sweep" and rng.random() < 0.4 else 0
    return _case(None, entry, n_side, cpd, clustered, softening, density, radius, record, slabs)


# ---------------------------------------------------------------- inputs

class _Positions:
    """A box as the library's Python binding takes it."""

    def __init__(self, cpd, x, y, z, cell_start):
        self.cpd, self.x, self.y, self.z, self.cell_start = cpd, x, y, z, cell_start
        self.n = int(cell_start[-1])

    def host(self):
        return _Positions(self.cpd, self.x.cpu().numpy(), self.y.cpu().numpy(),
                          self.z.cpu().numpy(), self.cell_start)


def _box(case, seed):
    _, synth = _package()
    x, y, z, cs = synth.clustered_box_device(
        case["n_side"] ** 3, case["cpd"], seed=seed, n_clumps=2000,
        clump_fraction=0.6 if case["clustered"] else 0.0)
    return _Positions(case["cpd"], x, y, z, cs)


def _seeds(case, seed):
    """One seed per box: two boxes are served, the others use one."""
    return [2 * seed + k for k in range(2 if case["entry"] == "serve" else 1)]


def _b2(case):
    return float(np.float32((0.2 / case["cpd"]) ** 2)) if case["density"] else 0.0


def _eps(case):
    _, synth = _package()
    return synth.kernel_eps(case["softening"], synth.plummer_eps(case["n_side"]))


def _config(case):
    capi, _ = _package()
    return dict(softening=case["softening"], eps=_eps(case), b2=_b2(case),
                near_field_radius=case["radius"],
                out_kind=capi.OUT_FLOAT4 if case["record"] == 4 else capi.OUT_FLOAT3)


def _slab_range(case):
    if not case["slabs"]:
        return 0, case["cpd"]
    lo = (case["cpd"] - case["slabs"]) // 2
    return lo, lo + case["slabs"]


def _requests(case, seed):
    """(box, slab) of the served requests: every slab of both boxes, in a seeded order."""
    k = np.random.default_rng(seed + 1000003).permutation(2 * case["cpd"])
    return [(int(i) // case["cpd"], int(i) % case["cpd"]) for i in k]


def _kick_inputs(case, n, seed):
    """Far-field accelerations and velocities, at the scale of the near field."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed * 31 + 5)
    far = torch.randn((n, 3), generator=g, device="cuda") * (0.1 * n)
    vel = torch.randn((n, 3), generator=g, device="cuda") * 1e-2
    return far, vel


def _kick_constants(case):
    """Output units of the raw kernel, and kicks that move velocities by a few per cent."""
    near = _eps(case) ** 1.5 if case["softening"] == SINGLE_SPLINE else 1.0
    n = case["n_side"] ** 3
    return dict(near_scale=near, rescale=-3.0 * 0.31 / (8 * math.pi * n), kick1=0.013,
                kick2=0.011, b2=_b2(case))


def _pinned(shape):
    return torch.empty(shape, dtype=torch.float32, pin_memory=True)


class State:
    """What a program holds between calls; frees the library's handles with it."""

    def __init__(self, case):
        self.case, self.closers = case, []

    def keep(self, thing):
        self.closers.append(thing)
        return thing

    def __del__(self):
        torch.cuda.synchronize()
        while self.closers:
            self.closers.pop().close()


def prepare(case, seed):
    capi, synth = _package()
    s = State(case)
    boxes = [_box(case, k) for k in _seeds(case, seed)]
    box = boxes[0]
    torch.cuda.synchronize()
    entry, w = case["entry"], case["record"]
    if entry == "driver":
        host = box.host()
        s.drv = s.keep(capi.Driver(
            host, softening=case["softening"], softening_length=synth.plummer_eps(case["n_side"]),
            near_field_radius=case["radius"], b2=_b2(case),
            out_kind=capi.OUT_FLOAT4 if w == 4 else capi.OUT_FLOAT3))
        # the AccSlabs in one arena
        s.acc = np.zeros((host.n, w), np.float32)
        for slab, (p0, p1) in enumerate(s.drv.slabs.ranges):
            s.drv.slabs.acc[slab] = s.acc[p0:p1]
            view = s.drv.slabs.view(slab)
            capi.check(capi.lib().nf_driver_set_slab(s.drv.h, slab, ctypes.byref(view)))
        return s
    if entry == "noalloc":
        s.cfg = capi.default_config(**_config(case))
        s.pos = torch.zeros((box.n, 4), device="cuda")
        s.pos[:, 0], s.pos[:, 1], s.pos[:, 2] = box.x, box.y, box.z
        s.cs = torch.from_numpy(box.cell_start).cuda()
        s.out = torch.empty((box.n, w), device="cuda")
        return s
    s.ctx = s.keep(capi.Context(**_config(case)))
    if entry == "timestep":
        s.box = box
        s.out = torch.empty((box.n, w), device="cuda")
        return s
    s.boxes = [s.keep(s.ctx.box(b)) for b in boxes]
    lo, hi = _slab_range(case)
    p0, p1 = s.boxes[0].slab_particles(lo, hi)
    if entry == "sweep":
        s.out = torch.empty((p1 - p0, w), device="cuda")
    elif entry == "kick":
        s.far, s.vel = _kick_inputs(case, box.n, seed)
        s.acc = torch.empty((box.n, w), device="cuda")
        s.stats = torch.empty((case["cpd"] ** 3, 3), device="cuda")
        s.k = _kick_constants(case)
    elif entry == "step":
        s.host = [_pinned(box.n) for _ in range(3)]
        for h, d in zip(s.host, (box.x, box.y, box.z)):
            h.copy_(d)
        s.out = _pinned((box.n, w))
    elif entry == "serve":
        s.out = [_pinned((b.n, w)) for b in boxes]
        s.requests = []
        for b, slab in _requests(case, seed):
            q0, q1 = s.boxes[b].slab_particles(slab, slab + 1)
            s.requests.append((s.boxes[b], slab, s.out[b].numpy()[q0:q1]))
        s.srv = s.keep(capi.Server(s.ctx))
    torch.cuda.synchronize()
    return s


def run(s):
    case = s.case
    entry = case["entry"]
    capi, _ = _package()
    if entry == "sweep":
        s.boxes[0].forces_device(*_slab_range(case), s.out.data_ptr())
        return s.out
    if entry == "kick":
        s.boxes[0].kick(0, case["cpd"], s.vel.data_ptr(), s.far.data_ptr(), s.acc.data_ptr(),
                        s.stats.data_ptr(), **s.k)
        return [s.acc, s.vel, s.stats]
    if entry == "step":
        s.boxes[0].step(*(h.numpy() for h in s.host), s.out.numpy())
        return s.out
    if entry == "timestep":
        box = s.ctx.box(s.box)
        box.forces_device(0, case["cpd"], s.out.data_ptr())
        box.close()
        return s.out
    if entry == "driver":
        pending = list(range(case["cpd"]))
        for slab in pending:
            s.drv.execute_slab(slab)
        while pending:
            for slab in list(pending):
                done = s.drv.slab_done(slab)
                if done < 0:
                    raise RuntimeError(capi.last_error())
                if done:
                    s.drv.finalize(slab)
                    pending.remove(slab)
            time.sleep(0)
        return s.acc
    if entry == "serve":
        tickets = [s.srv.submit(b, slab, o) for b, slab, o in s.requests]
        for t in tickets:
            s.srv.wait(t)
        return s.out
    capi.check(capi.lib().nf_forces_noalloc(
        ctypes.byref(s.cfg), case["cpd"], s.pos.data_ptr(), s.cs.data_ptr(), 0, case["cpd"],
        s.out.data_ptr(), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)),
        "nf_forces_noalloc")
    return s.out


def _pair_estimate(case):
    """Pairs of one pass.  Uniform: the mean occupancy.  Clustered: a particle also meets its
    own clump, 4.2e-4 of all particles in the mean over the generator's clump masses (exact to
    some per cent for a whole box)."""
    n, w = case["n_side"] ** 3, 2 * case["radius"] + 1
    per_sink = w ** 3 * n / case["cpd"] ** 3 + (4.2e-4 * n if case["clustered"] else 0.0)
    share = case["slabs"] / case["cpd"] if case["slabs"] else 1.0
    return n * per_sink * share * (2 if case["entry"] == "serve" else 1)


#: flops of one pair interaction (an FMA counts two, rsqrt one, one Newton step included)
PAIR_FLOPS = {PLUMMER: 23, SINGLE_SPLINE: 24, CUBIC_SPLINE: 38, CUBIC_PLUMMER: 26}


def work(case):
    n = case["n_side"] ** 3
    per = 12 + 4 * case["record"]
    if case["entry"] == "kick":
        per += 12 + 24
    if case["entry"] == "serve":
        n = 2 * n
    elif case["slabs"]:
        n = n * case["slabs"] / case["cpd"]
    flops = PAIR_FLOPS[case["softening"]] + (4 if case["density"] else 0)
    return {"bytes": float(n * per), "flops": float(_pair_estimate(case) * flops)}


def tolerance(case):
    return {"rel": 4e-6, "max": 1e-4}


# ---------------------------------------------------------------- 64-bit reference

#: pairs up to which the direct sum in 64 bits takes under about 20 seconds
EXACT_PAIRS = 3e10


def _force64(softening, eps, r2):
    """f(r^2) of the output sum f (sink - source), the softening kernels' definitions."""
    if softening == PLUMMER:
        return (r2 + eps) ** -1.5
    if softening == SINGLE_SPLINE:  # eps = 1/e^2, f in units of e^-3
        u2 = torch.clamp(r2 * eps, min=1e-40)
        u = torch.sqrt(u2)
        return torch.where(u2 > 1, u ** -3, -15 * u + 6 * u2 + 10)
    r = torch.sqrt(torch.clamp(r2, min=1e-40))
    if softening == CUBIC_SPLINE:  # eps = 1/e
        u = r * eps
        far = r ** -3
        mid = far * (-1 / 15 + u ** 3 * (8 / 3 - 3 * u + 1.2 * u ** 2 - u ** 3 / 6))
        near = eps ** 3 * (4 / 3 - 1.2 * u ** 2 + 0.5 * u ** 3)
        return torch.where(u >= 2, far, torch.where(u >= 1, mid, near))
    return 1.0 / (r ** 3 + eps)  # eps = e^3


def _direct64(box, softening, eps, b2, R, lo, hi):
    """Accelerations (and density sum) of slabs [lo, hi) in 64 bits, plain torch: cell by cell,
    every sink against all particles of the (2R+1)^3 cells around its cell.  The columns of
    cells carry R ghost cells at both ends, so that a column's sources are one run."""
    dev, cpd = box.x.device, box.cpd
    h = 1.0 / cpd
    cs = np.asarray(box.cell_start)
    xyz = torch.stack([box.x, box.y, box.z], 1).double()
    out = torch.zeros((int(cs[hi * cpd * cpd] - cs[lo * cpd * cpd]), 4), dtype=torch.float64,
                      device=dev)
    W = 2 * R + 1
    zz = np.arange(-R, cpd + R)
    dz_all = torch.from_numpy(zz * h).to(dev)
    for x in range(lo, hi):
        for y in range(cpd):
            # the W x W columns around (x, y): their particles in z order, ghosts included
            starts, counts, shifts = [], [], []
            for dx in range(-R, R + 1):
                for dy in range(-R, R + 1):
                    c = (((x + dx) % cpd) * cpd + (y + dy) % cpd) * cpd + zz % cpd
                    starts.append(cs[c])
                    counts.append(cs[c + 1] - cs[c])
                    shifts.append((dx * h, dy * h))
            starts, counts = np.stack(starts), np.stack(counts)       # (columns, z)
            # order by z cell first: a sink cell then meets W consecutive z layers
            st, ct = starts.T.ravel(), counts.T.ravel()
            first = np.concatenate([[0], np.cumsum(ct)])
            layer = first[::W * W]                                    # start of each z layer
            ct_d = torch.from_numpy(ct).to(dev)
            run_of = torch.repeat_interleave(torch.arange(len(ct), device=dev), ct_d)
            idx = torch.from_numpy(st - first[:-1]).to(dev)[run_of] + torch.arange(
                int(first[-1]), device=dev)
            src = xyz[idx]
            sh = torch.tensor(shifts, dtype=torch.float64, device=dev)
            col = run_of % (W * W)
            src[:, :2] += sh[col]
            src[:, 2] += dz_all[run_of // (W * W)]
            base = (x * cpd + y) * cpd
            for z in range(cpd):
                a, b = int(cs[base + z]), int(cs[base + z + 1])
                q = src[int(layer[z]):int(layer[z + W])]
                if a == b:
                    continue
                for a0 in range(a, b, max(1, int(2e8 // max(len(q), 1)))):
                    a1 = min(b, a0 + max(1, int(2e8 // max(len(q), 1))))
                    p = xyz[a0:a1].clone()
                    p[:, 2] += z * h
                    d = p.T[:, :, None] - q.T[:, None, :]
                    r2 = (d * d).sum(0)
                    o = out[a0 - int(cs[lo * cpd * cpd]):a1 - int(cs[lo * cpd * cpd])]
                    f = _force64(softening, eps, r2)
                    o[:, :3] = torch.einsum("ij,cij->ic", f, d)
                    if b2:
                        o[:, 3] = torch.clamp(b2 - r2, min=0).sum(1)
    return out


def _exact_pairs(box, R):
    """Pairs of the whole box, exactly."""
    c = torch.from_numpy(np.diff(box.cell_start).reshape((box.cpd,) * 3)).double()
    s = c
    for axis in range(3):
        s = sum(torch.roll(s, k, axis) for k in range(-R, R + 1))
    return float((c * s).sum())


def exact(case, seed):
    boxes = [_box(case, k) for k in _seeds(case, seed)]
    lo, hi = _slab_range(case)
    share = (hi - lo) / case["cpd"]
    if sum(_exact_pairs(b, case["radius"]) for b in boxes) * share > EXACT_PAIRS:
        return None
    eps = float(np.float32(_eps(case)))
    args = (case["softening"], eps, _b2(case), case["radius"])
    w = case["record"]
    if case["entry"] == "serve":
        return [_direct64(b, *args, lo, hi)[:, :w].cpu() for b in boxes]
    box = boxes[0]
    acc = _direct64(box, *args, lo, hi)
    if case["entry"] != "kick":
        return acc[:, :w].cpu()
    k = _kick_constants(case)
    far, vel = _kick_inputs(case, box.n, seed)
    a = (acc[:, :3] * float(np.float32(k["near_scale"])) + far.double()) * k["rescale"]
    v = vel.double() + a * k["kick1"]
    cnt = torch.from_numpy(np.diff(box.cell_start)).cuda()
    cell = torch.repeat_interleave(torch.arange(len(cnt), device="cuda"), cnt)
    stats = torch.zeros((len(cnt), 3), dtype=torch.float64, device="cuda")
    stats[:, 0].index_add_(0, cell, (v * v).sum(1))
    stats[:, 0] /= torch.clamp(cnt, min=1)
    for i, q in ((1, v), (2, a)):
        stats[:, i] = torch.zeros_like(stats[:, i]).scatter_reduce_(
            0, cell, q.abs().amax(1), "amax")
    rec = torch.cat([a, (acc[:, 3:] - k["b2"])], 1)[:, :w]
    return [rec, v + a * k["kick2"], stats]
