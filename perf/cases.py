"""The estimation epoch's workloads, as a user's program calls them.

Each case is a seeded synthetic heart (a cuboid or an ellipsoidal shell with a pathological block),
its ground-truth measurements with 1 % noise, and one call of the public API: an epoch whose model
stays on the device, an epoch on a model in host memory, the forward simulation, the scenario loop,
or a batched epoch. The ranges are those of the repository's own workloads: voxel edges of 2.0, 2.5
and 5.0 mm, 64 to 47,264 voxels, beats of 100 to 4,000 steps at 2 kHz, 1 to 3 beats, 37 to 256
triaxial sensors, SGD and Adam, both all-pass derivatives, gains alone or gains and delays trained.
"""

import math

import numpy as np
import torch

from cardiotrust_b200 import algorithm as alg
from cardiotrust_b200 import scenario as sc

_BASE = dict(kind="epoch", mask="cuboid", nx=8, ny=8, nz=8, voxel_mm=2.5, steps=500, beats=1, sensors=37, patho=3,
             grad="reference", precision="bf16x6", optimizer="sgd", lr=0.5, derivative="textbook", delays=True,
             batch_size=0, epochs=1, members="")


def listed():
    def case(name, **kw):
        return dict(_BASE, name=name, **kw)

    return [
        # the smallest calls: an interactive run on a coarse 5 mm model, gains only (the config's defaults)
        case("epoch_tiny", nx=4, ny=4, nz=4, voxel_mm=5.0, steps=300, patho=2, delays=False),
        # the plain config: 512 voxels, half-second beat
        case("epoch_cuboid8", optimizer="adam", lr=1e-3),
        # the headline workload: 8,000 voxels, one-second beat
        case("epoch_cuboid20", nx=20, ny=20, nz=20, steps=2000, patho=5, optimizer="adam", lr=1e-3),
        # the same for a program that keeps the model in (pinned) host memory
        case("host_cuboid20", kind="host", nx=20, ny=20, nz=20, steps=2000, patho=5),
        # exact gradients on the headline workload
        case("adjoint_cuboid20", nx=20, ny=20, nz=20, steps=2000, patho=5, grad="adjoint", lr=5e-3),
        # the full-size ventricular shell, two-second beat, exact gradients: the largest call
        case("adjoint_shell64", mask="shell", nx=64, ny=64, nz=48, steps=4000, patho=8, grad="adjoint", lr=5e-3),
        # several beats with an update every second one, simple derivative, FP32 products, 2 mm voxels
        case("epoch_beats", mask="shell", nx=33, ny=31, nz=25, voxel_mm=2.0, steps=1500, beats=3, batch_size=2, patho=6,
             derivative="simple", precision="fp32"),
        # a dense sensor array: 768 rows, odd grid
        case("epoch_sensors256", nx=16, ny=15, nz=17, steps=1500, sensors=256),
        # ground-truth simulation on the full-size shell
        case("simulate_shell64", kind="simulate", mask="shell", nx=64, ny=64, nz=48, steps=1000),
        # the whole scenario loop on a small model, exact gradients
        case("loop_cuboid9", kind="loop", nx=9, ny=8, nz=7, steps=500, grad="adjoint", lr=5e-3, delays=False, epochs=10),
        # parameter studies: scenarios of uneven size in one schedule
        case("batch_adjoint", kind="batch", grad="adjoint", lr=5e-3, patho=5,
             members="cuboid 9x8x9 1000 2 37;shell 22x22x17 1500 1 64;cuboid 17x13x15 1200 2 45;"
                     "shell 32x32x24 1300 1 37;cuboid 22x21x20 1100 1 90;cuboid 27x25x26 1300 1 51"),
        case("batch_reference", kind="batch",
             members="cuboid 8x8x8 500 1 37;cuboid 7x9x10 700 2 37;shell 16x16x12 600 1 40;cuboid 11x10x12 800 1 37"),
    ]


def _member(case, text):
    mask, shape, steps, beats, sensors = text.split()
    nx, ny, nz = (int(n) for n in shape.split("x"))
    return dict(case, kind="epoch", mask=mask, nx=nx, ny=ny, nz=nz, steps=int(steps), beats=int(beats),
                sensors=int(sensors), members="")


def _members(case):
    """The single-scenario cases that a case is made of."""
    if case["kind"] != "batch":
        return [case]
    return [_member(case, t) for t in case["members"].split(";")]


def _spec(case, seed):
    shape = (case["nx"], case["ny"], case["nz"])
    f = case["nx"] / 64.0
    return sc.ScenarioSpec(shape=shape, mask=case["mask"], shell_semi_axes=(30.0 * f, 25.0 * f, 22.0 * f),
                           shell_thickness=max(2.0, 8.0 * f), voxel_size_mm=case["voxel_mm"],
                           num_steps=case["steps"], num_beats=case["beats"], num_sensors=case["sensors"],
                           patho_size=case["patho"], noise_fraction=0.01, seed=int(seed) % (1 << 31))


def _travel(mask, shape, voxel_mm):
    """Steps in which a pulse starts and its activation crosses the grid (0.6 m/s, 2 kHz)."""
    return 150 + int(sum(shape) * (1.8 if mask == "shell" else 1.2) * voxel_mm / 0.6 * 2.0)


def draw(rng):
    def log(a, b):
        return math.exp(rng.uniform(math.log(a), math.log(b)))

    def grid(most):
        mask = rng.choice(["cuboid", "cuboid", "shell"])
        v = log(64, most)
        if mask == "shell":
            f = (max(v, 700.0) / 47264.0) ** (1.0 / 3.0)
            return mask, (math.ceil(64 * f), math.ceil(64 * f), math.ceil(48 * f))
        e = v ** (1.0 / 3.0)
        nx, ny = (max(4, round(e * rng.uniform(0.8, 1.25))) for _ in range(2))
        return mask, (nx, ny, max(4, round(v / (nx * ny))))

    c = dict(_BASE, kind=rng.choice(["epoch", "epoch", "epoch", "host", "simulate", "loop", "batch"]))
    most = {"loop": 2000, "batch": 12000}.get(c["kind"], 30000)
    c["grad"] = rng.choice(["reference", "adjoint"])
    c["lr"] = 5e-3 if c["grad"] == "adjoint" else 0.5
    if c["kind"] == "batch":
        texts = []
        for _ in range(rng.randint(2, 6)):
            mask, shape = grid(most)
            low = _travel(mask, shape, 2.5)
            texts.append("%s %s %d %d %d" % (mask, "x".join(map(str, shape)), log(low, max(2 * low, 1500)),
                                             rng.randint(1, 2), rng.randint(37, 128)))
        c["members"] = ";".join(texts)
        return c
    c["voxel_mm"] = rng.choice([2.0, 2.5, 2.5, 5.0])
    c["mask"], (c["nx"], c["ny"], c["nz"]) = grid(most if c["voxel_mm"] < 5.0 else 4000)
    low = _travel(c["mask"], (c["nx"], c["ny"], c["nz"]), c["voxel_mm"])
    c["steps"] = int(log(low, max(3000, 1.5 * low) if c["kind"] != "loop" else 2 * low))
    c["beats"] = rng.choice([1, 1, 2, 3]) if c["nx"] * c["ny"] * c["nz"] < 4000 else 1
    c["sensors"] = int(log(37, 256)) if c["kind"] != "loop" else 37
    c["patho"] = max(2, min(c["nx"], c["ny"], c["nz"]) // 4)
    c["derivative"] = rng.choice(["textbook", "textbook", "simple"])
    c["delays"] = rng.random() < 0.7
    c["precision"] = "fp32" if rng.random() < 0.15 else "bf16x6"
    c["epochs"] = rng.randint(2, 8) if c["kind"] == "loop" else 1
    return c


# ---------------------------------------------------------------------------------------------
# inputs


_CTX = None


def _context():
    global _CTX
    if _CTX is None:
        _CTX = alg.Context(0)
    return _CTX


class _Plain:
    """The state recursion on plain torch tensors: inputs, delays and gains of one parameter set."""

    def __init__(self, p, H, ctrl, u, dtype):
        dev = "cuda"
        self.V = p.coefs.shape[0]
        self.osi = torch.from_numpy(np.ascontiguousarray(p.output_state_indices)).to(dev)[::3].long()  # [V,78]
        self.valid = (self.osi >= 0).to(dtype)
        self.g = torch.from_numpy(p.gains).to(dev, dtype).view(self.V, 3, 78)
        self.H = torch.from_numpy(np.ascontiguousarray(H)).to(dev, dtype)
        self.ctrl = torch.from_numpy(ctrl).to(dev, dtype)
        self.u = torch.from_numpy(u).to(dev, dtype)
        self.T, self.S, self.dtype = u.shape[0], 3 * self.V, dtype
        self.set(torch.from_numpy(p.coefs).to(dev, dtype), torch.from_numpy(p.delays).to(dev))

    def set(self, coefs, delays):
        self.coefs, self.delays = coefs, delays.long()
        self.c = coefs.repeat_interleave(3, 1)  # [V,78]
        self.d = self.delays.repeat_interleave(3, 1)
        conn = self.osi >= 0
        self.pad = int(self.d[conn].max()) + 1 if bool(conn.any()) else 1
        j = self.osi.clamp(min=0)
        # x[t-d, j] of the history stored from row `pad` on; absent neighbours read a zero row
        self.at = torch.where(conn, (self.pad - self.d) * self.S + j, torch.zeros_like(j))
        self.step = torch.where(conn, torch.full_like(j, self.S), torch.zeros_like(j))

    def states(self):
        X = torch.zeros((self.pad + self.T, self.S), device="cuda", dtype=self.dtype)
        flat, at = X.view(-1), self.at.clone()
        ap = torch.zeros((self.V, 78), device="cuda", dtype=self.dtype)
        last = torch.zeros_like(ap)
        gt = (self.g * self.valid[:, None, :]).contiguous()
        drive = self.u[:, None] * self.ctrl[None, :] if self.T * self.S < 1e8 else None
        for t in range(self.T):
            inp = flat[at]
            at += self.step
            ap = torch.addcmul(last, self.c, inp - ap)
            last = inp
            x = torch.bmm(gt, ap[:, :, None]).view(-1)
            X[self.pad + t] = x + (drive[t] if drive is not None else self.u[t] * self.ctrl)
        return X[self.pad:]


def _scenario(case, seed):
    """The built scenario with its noisy ground-truth measurements."""
    scn = sc.build(_spec(case, seed), _context())
    if case["kind"] == "simulate":
        return scn
    plain = _Plain(scn.truth, scn.measurement_matrix, scn.control_matrix, scn.control_function, torch.float32)
    X = plain.states().double()
    y = torch.stack([X @ h.double().T for h in plain.H])  # [B,T,M]
    gen = torch.Generator("cuda").manual_seed(int(seed) + 7919)
    y = y + torch.randn(y.shape, generator=gen, device="cuda", dtype=torch.float64) * (0.01 * y.square().mean().sqrt())
    scn.measurements = y.float().cpu().numpy()
    return scn


def _algorithm(case):
    return alg.Algorithm(optimizer=alg.Optimizer.Adam if case["optimizer"] == "adam" else alg.Optimizer.Sgd,
                         learning_rate=case["lr"], batch_size=case["batch_size"], epochs=case["epochs"],
                         freeze_delays=not case["delays"],
                         ap_derivative=alg.APDerivative.Simple if case["derivative"] == "simple"
                         else alg.APDerivative.Textbook)


def _slots(case):
    if case["kind"] == "loop":
        return case["epochs"]
    return -(-case["beats"] // case["batch_size"]) if case["batch_size"] else 1


def _pinned(shape, dtype=torch.float32):
    return torch.zeros(shape, dtype=dtype, pin_memory=True).numpy()


def _engine(case, scn):
    return alg.EpochEngine.from_scenario(_context(), scn, truth=case["kind"] == "simulate",
                                         num_batch_slots=_slots(case), algorithm=_algorithm(case))


def prepare(case, seed):
    grad = alg.GradMode.Adjoint if case["grad"] == "adjoint" else alg.GradMode.Reference
    prec = alg.Precision.Fp32 if case["precision"] == "fp32" else alg.Precision.Bf16x6
    s = dict(kind=case["kind"], grad=grad, prec=prec, out=[], engines=[])
    for i, c in enumerate(_members(case)):
        scn = _scenario(c, seed + 1000 * i)
        e = _engine(c, scn)
        s["engines"].append(e)
        V, S = e.dims["V"], e.dims["S"]
        s["out"].append(dict(gains=_pinned((S, 78)), coefs=_pinned((V, 26))))
        s["order"] = np.arange(c["beats"], dtype=np.int32)
        if case["kind"] == "host":
            o = s["out"][0]
            o["gains"][:], o["coefs"][:] = scn.model.gains, scn.model.coefs
            o["delays"] = _pinned((V, 26), torch.int32)
            o["delays"][:] = scn.model.delays
            o["loss_batch"] = _pinned((_slots(c),))
            s["measurements"] = _pinned(scn.measurements.shape)
            s["measurements"][:] = scn.measurements
    if case["kind"] == "loop":
        s["orders"] = np.tile(s["order"], (case["epochs"], 1))
    if case["kind"] == "batch":
        s["batch"] = alg.EpochBatch(_context(), s["engines"], grad_mode=grad, precision=prec)
    return s


def _read_gradients(e, o):
    return dict(grad_gains=e.read_into("grad_gains", o["gains"]), grad_coefs=e.read_into("grad_coefs", o["coefs"]),
                loss_batch=e.read("loss_batch"))


def run(s):
    e, o = s["engines"][0], s["out"][0]
    if s["kind"] == "simulate":
        return e.simulate()
    if s["kind"] == "host":
        e.run_epoch_host(0, o["gains"], o["coefs"], o["delays"], measurements=s["measurements"],
                         loss_batch=o["loss_batch"], beat_order=s["order"], grad_mode=s["grad"], precision=s["prec"])
        return o
    if s["kind"] == "loop":
        _, losses, _ = e.run_model_based(0, beat_orders=s["orders"], grad_mode=s["grad"], precision=s["prec"])
        return dict(losses=losses, gains=e.read_into("gains", o["gains"]), coefs=e.read_into("coefs", o["coefs"]))
    if s["kind"] == "batch":
        s["batch"].batch_indices[:] = 0
        s["batch"].run_epoch()
        return [_read_gradients(m, q) for m, q in zip(s["engines"], s["out"])]
    e.run_epoch(0, beat_order=s["order"], grad_mode=s["grad"], precision=s["prec"])
    return _read_gradients(e, o)


def work(case):
    """Operations of the recursion, the products and the derivation; parameters, lead field,
    measurements and gradients once, and the states and mapped residuals of every step once."""
    total = dict(bytes=0.0, flops=0.0)
    for c in _members(case):
        V = sc.voxel_count(_spec(c, 0))
        n, T, M, B = c["epochs"], c["steps"], 3 * c["sensors"], c["beats"]
        steps = float(n) * V * T * B
        total["flops"] += steps * (78 * 3 + 234 * 2) + n * 2.0 * M * 3 * V * T * B
        total["bytes"] += 4.0 * n * (3 * V * 78 + 2 * V * 26 + B * M * 3 * V + B * T * M + 3 * V * T * B)
        if c["kind"] != "simulate":
            total["flops"] += n * 2.0 * M * 3 * V * T * B
            # per voxel-step: reference 234 gain terms (and 234 coefficient terms), or the adjoint recursion
            per = (78 * 3 + 234 * 2) + 78 * 6 + 234 * 4 if c["grad"] == "adjoint" else 78 * 3 + 234 * 2 + 234 * 4 * c["delays"]
            total["flops"] += steps * per
            total["bytes"] += 4.0 * n * (3 * V * T * B + 2 * (3 * V * 78 + V * 26))
    return total


# ---------------------------------------------------------------------------------------------
# the same in 64 bits, on plain torch tensors


def _epoch64(m, z, case, adjoint):
    """One epoch of `m` (updated in place; SGD): (dG, dC, loss_batch)."""
    T, V, M = m.T, m.V, m.H.shape[1]
    thr, ms = float(np.float32(1.01)), 1.0 / M
    bs = case["batch_size"]
    zero = lambda: (torch.zeros((V, 3, 78), device="cuda", dtype=torch.float64),  # noqa: E731
                    torch.zeros((V, 78), device="cuda", dtype=torch.float64),
                    torch.zeros((V, 78), device="cuda", dtype=torch.float64),
                    torch.zeros((V, 78), device="cuda", dtype=torch.float64), 0.0)
    dG, dC, fir, iir, reg = zero()
    losses, beats = [], 0

    def finish(n):
        losses.append((reg_t + mse).mean())
        rate = case["lr_now"] / float(T * n)
        m.g = m.g - rate * dG
        if case["delays"]:
            m.coefs = m.coefs - rate * dC.view(V, 26, 3).sum(2)
            m.set(m.coefs, m.delays)

    for beat in range(case["beats"]):
        X = m.states()
        R = X @ m.H[beat].T - z[beat]
        mse = R.square().sum(1) / M
        MR = R @ m.H[beat]
        x3 = X.view(T, V, 3)
        over = x3.abs().sum(2) - thr
        f = over.clamp(min=0)
        reg_t = reg + f.square().sum(1).cumsum(0)
        reg = reg_t[-1]
        pull = (f[:, :, None] * torch.sign(x3)).view(T, -1)
        q = ms * MR + pull  # [T,S]
        pad = torch.cat([torch.zeros((m.pad, m.S), device="cuda", dtype=torch.float64), X])
        valid = m.valid
        if adjoint:
            # lx backwards in time, gathered by the source of every item, then the forward sweep of the gradients
            L = torch.zeros((T + m.pad, m.S), device="cuda", dtype=torch.float64)
            lap = torch.zeros((V, 78), device="cuda", dtype=torch.float64)
            box = torch.zeros((m.pad + 1, m.S), device="cuda", dtype=torch.float64)
            gt = (m.g * valid[:, None, :]).transpose(1, 2).contiguous()
            n = m.pad + 1
            flat = box.view(-1)
            tgt = m.osi.clamp(min=0)
            for t in range(T - 1, -1, -1):
                lx = q[t] + box[t % n]
                box[t % n] = 0
                L[t] = lx
                new = torch.bmm(gt, lx.view(V, 3, 1)).view(V, 78) - m.c * lap
                w = (m.c * new + lap) * valid
                row = (t - m.d) % n
                w = torch.where(t - m.d >= 0, w, torch.zeros_like(w))
                flat.scatter_add_(0, (row * m.S + tgt).view(-1), w.view(-1))
                lap = new
            q = L[:T]
        ap = torch.zeros((V, 78), device="cuda", dtype=torch.float64)
        last, tan = torch.zeros_like(ap), torch.zeros_like(ap)
        flat, at = pad.view(-1), m.at.clone()
        for t in range(T):
            inp = flat[at]
            at += m.step
            before = ap
            ap = torch.addcmul(last, m.c, inp - ap)
            qt = q[t].view(V, 3, 1)
            dG.addcmul_(qt, (ap * valid)[:, None, :])
            if case["delays"]:
                mr = (q if adjoint else ms * MR)[t].view(V, 3, 1)
                gm = (m.g * mr).sum(1) * valid
                if adjoint:
                    tan = (inp - before) - m.c * tan
                    dC.addcmul_(gm, tan)
                elif case["derivative"] == "textbook":
                    on = t >= m.d
                    fir = torch.where(on, inp - m.c * fir, fir)
                    iir = torch.where(on, before - m.c * iir, iir)
                    dC.addcmul_(gm, fir - iir)
                else:
                    dC.addcmul_(gm, torch.where(t >= m.d, inp - before, torch.zeros_like(ap)))
            last = inp
        beats += 1
        if bs and beats == bs:
            finish(beats)
            dG, dC, fir, iir, reg = zero()
            beats = 0
    if not bs or beats:
        finish(beats)
    return dG, dC.view(V, 26, 3).sum(2), torch.stack(losses), reg_t + mse, mse, reg_t


def exact(case, seed):
    out = []
    for i, c in enumerate(_members(case)):
        scn = _scenario(c, seed + 1000 * i)
        p = scn.truth if c["kind"] == "simulate" else scn.model
        m = _Plain(p, scn.measurement_matrix, scn.control_matrix, scn.control_function, torch.float64)
        if c["kind"] == "simulate":
            X = m.states()
            return torch.stack([X @ h.T for h in m.H])
        if c["delays"] and c["kind"] == "loop":
            return None  # the coefficients may cross into the next integer delay
        z = torch.from_numpy(scn.measurements).to("cuda", torch.float64)
        losses = []
        for k in range(c["epochs"]):
            # the scenario loop's first epoch has the learning rate 0
            c["lr_now"] = 0.0 if c["kind"] == "loop" and k == 0 else c["lr"]
            dG, dC, loss, per, mse, reg = _epoch64(m, z, c, c["grad"] == "adjoint")
            losses.append(torch.stack([loss[-1], mse.mean(), reg.mean()]))
        if c["kind"] == "loop":
            out.append(dict(losses=torch.stack(losses), gains=m.g.reshape(-1, 78), coefs=m.coefs))
        elif c["kind"] == "host":
            out.append(dict(gains=m.g.reshape(-1, 78), coefs=m.coefs, delays=None, loss_batch=loss))
        else:
            out.append(dict(grad_gains=dG.reshape(-1, 78), grad_coefs=dC if c["delays"] else None, loss_batch=loss))
    return out if case["kind"] == "batch" else out[0]
