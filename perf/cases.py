"""Performance cases of the hard-disk engine: what a user's program has it do, through the public entry points.

A case is a dict of plain values:
  kind     serial    restart from host state, `coll` collisions per system in the serial-exact engine, state back
           rounds    restart from host state, one system to time `t` in the round engine (exact mode), state back
           growth    new systems of growing disks up to the growth stop (the drop-in program's default start), state back
           tangent   restart, `k` tangent vectors over `coll` collisions, re-orthonormalised every `qr`: Lyapunov exponents
           gradient  restart, final mean-square displacement after `coll` collisions and its gradient, checkpoints every `ckpt`
           sample    what happens at a sampling point: every disk free-flown, state back, g(r) of the system
  systems  independent systems of one context;  disks, disks_min: largest and smallest of them
  phi      packing fraction of the lattice of unit disks;  mix: half of the disks have radius 0.714 and mass 0.51

Starts are triangular lattices with every disk displaced inside its free space and normally distributed velocities
(zero momentum, one unit of energy per disk).
"""
import heapq
import math

import numpy as np

import __graft_entry__ as entry

edmd = entry._load("edmd")


def listed():
    return [
        # one small box for a few collisions: an interactive step, or one evaluation inside an optimiser's loop
        {"name": "serial_one", "kind": "serial", "systems": 1, "disks": 203, "disks_min": 203, "phi": 0.60, "mix": False, "coll": 150},
        # an ensemble of mixed boxes, more of them than the GPU holds at once: parameter studies in bidisperse disks
        {"name": "serial_batch", "kind": "serial", "systems": 2600, "disks": 1024, "disks_min": 64, "phi": 0.55, "mix": True, "coll": 1200},
        # a large ensemble of very small boxes: the thread-per-system engine's range
        {"name": "serial_many", "kind": "serial", "systems": 16384, "disks": 96, "disks_min": 96, "phi": 0.55, "mix": False, "coll": 150},
        # the default start of the drop-in program, for an ensemble
        {"name": "growth_batch", "kind": "growth", "systems": 192, "disks": 257, "disks_min": 129, "phi": 0.50, "mix": True},
        # the plain system of the reference's command line
        {"name": "rounds_2k", "kind": "rounds", "systems": 1, "disks": 1980, "disks_min": 1980, "phi": 0.70, "mix": False, "t": 1.3},
        # a system of the size of published melting studies, bidisperse
        {"name": "rounds_60k", "kind": "rounds", "systems": 1, "disks": 60001, "disks_min": 60001, "phi": 0.74, "mix": True, "t": 1.2},
        # one very large system
        {"name": "rounds_1m", "kind": "rounds", "systems": 1, "disks": 1000000, "disks_min": 1000000, "phi": 0.72, "mix": False, "t": 0.7},
        # the largest one, dense
        {"name": "rounds_4m", "kind": "rounds", "systems": 1, "disks": 4000000, "disks_min": 4000000, "phi": 0.78, "mix": False, "t": 0.3},
        # Lyapunov spectrum of one system, and of an ensemble
        {"name": "tangent_one", "kind": "tangent", "systems": 1, "disks": 1024, "disks_min": 1024, "phi": 0.60, "mix": False,
         "coll": 800, "k": 32, "qr": 100},
        {"name": "tangent_batch", "kind": "tangent", "systems": 128, "disks": 512, "disks_min": 384, "phi": 0.60, "mix": False,
         "coll": 400, "k": 16, "qr": 100},
        # gradients of the final mean-square displacement for an ensemble
        {"name": "gradient_batch", "kind": "gradient", "systems": 96, "disks": 512, "disks_min": 320, "phi": 0.60, "mix": True,
         "coll": 400, "ckpt": 100},
        # a sampling point of a medium system
        {"name": "sample", "kind": "sample", "systems": 1, "disks": 100001, "disks_min": 100001, "phi": 0.70, "mix": False,
         "dr": 0.05, "max_r": 10.0},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["serial", "serial", "rounds", "rounds", "growth", "tangent", "gradient", "sample"])
    phi = round(rng.uniform(0.30, 0.75), 3)
    mix = rng.random() < 0.5
    if kind == "serial":
        if rng.random() < 0.3:                      # the thread-per-system engine's range
            n = rng.randint(16384, 20000)
            top = rng.randint(33, 96)
            return {"kind": kind, "systems": n, "disks": top, "disks_min": top, "phi": phi, "mix": mix, "coll": rng.randint(40, 150)}
        n = _log(rng, 1, 3000)
        top = _log(rng, 64, 1024)
        return {"kind": kind, "systems": n, "disks": top, "disks_min": rng.randint(max(33, top // 16), top), "phi": phi, "mix": mix,
                "coll": rng.randint(100, 1200)}
    if kind == "rounds":
        n = _log(rng, 500, 1500000)
        t = min(1.5, 1.0e6 / n)
        return {"kind": kind, "systems": 1, "disks": n, "disks_min": n, "phi": round(rng.uniform(0.45, 0.78), 3), "mix": mix,
                "t": round(t * rng.uniform(0.4, 0.8), 3)}
    if kind == "growth":
        top = _log(rng, 40, 300)
        return {"kind": kind, "systems": _log(rng, 1, 192), "disks": top, "disks_min": rng.randint(top // 2, top),
                "phi": round(rng.uniform(0.30, 0.60), 3), "mix": True}
    n = 1 if rng.random() < 0.4 else _log(rng, 2, 128)
    top = _log(rng, 128, 512 if n > 1 else 2000)
    low = rng.randint(top // 2, top) if n > 1 else top
    if kind == "tangent":
        return {"kind": kind, "systems": n, "disks": top, "disks_min": low, "phi": phi, "mix": mix, "coll": rng.randint(100, 400),
                "k": rng.randint(1, 32), "qr": rng.choice([25, 50, 100])}
    if kind == "gradient":
        return {"kind": kind, "systems": n, "disks": top, "disks_min": low, "phi": phi, "mix": mix, "coll": rng.randint(100, 400),
                "ckpt": rng.choice([50, 100, 150])}
    n = _log(rng, 1000, 200000)
    return {"kind": "sample", "systems": 1, "disks": n, "disks_min": n, "phi": round(rng.uniform(0.45, 0.78), 3), "mix": mix,
            "dr": rng.choice([0.02, 0.05, 0.1]), "max_r": round(rng.uniform(3.0, 10.0), 2)}


# ------------------------------------------------------------------ starts

def _sizes(case):
    """Disks of every system: at most 24 different sizes, spread evenly over the case's range."""
    n, lo, hi = case["systems"], case["disks_min"], case["disks"]
    d = max(1, min(n, 24))
    values = [hi] if d == 1 or lo == hi else [lo + (hi - lo) * k // (d - 1) for k in range(d)]
    return [values[s % len(values)] for s in range(n)]


def _starts(case, seed):
    """Start states of the case's systems, as arrays of the host: one dict per group of systems of one size."""
    sizes = _sizes(case)
    groups = []
    for size in sorted(set(sizes)):
        rng = np.random.default_rng([seed, size])
        count = sizes.count(size)
        rows = max(2, int(math.sqrt(size * 2 / math.sqrt(3.0)) / 2 + 0.5) * 2)
        cols = -(-size // rows)
        a = math.sqrt(2.0 * math.pi / (math.sqrt(3.0) * case["phi"]))       # lattice constant of unit disks
        Lx, Ly = cols * a, rows * a * math.sqrt(3.0) / 2
        site = np.arange(rows * cols)
        keep = np.sort(rng.permutation(site)[:size])
        gx, gy = keep % cols, keep // cols
        free = 0.49 * (a - 2.0)
        r = free * np.sqrt(rng.random((count, size)))
        w = rng.random((count, size)) * (2 * math.pi)
        x = np.mod((gx + 0.5 * (gy % 2)) * a + r * np.cos(w), Lx)
        y = np.mod(gy * (Ly / rows) + r * np.sin(w), Ly)
        x[x >= Lx] = 0.0
        y[y >= Ly] = 0.0
        rad = np.ones((count, size))
        m = np.ones((count, size))
        if case["mix"]:
            small = rng.random((count, size)) < 0.5
            rad[small] = 0.714
            m[small] = 0.51
        vx, vy = rng.standard_normal((2, count, size)) / np.sqrt(m)
        for v in (vx, vy):
            v -= (v * m).sum(1, keepdims=True) / m.sum(1, keepdims=True)
        scale = np.sqrt(0.5 * (m * (vx * vx + vy * vy)).sum(1, keepdims=True) / size)
        groups.append(dict(N=size, Lx=Lx, Ly=Ly, x=x, y=y, vx=vx / scale, vy=vy / scale, rad=rad, m=m))
    # in system order
    taken = {g["N"]: 0 for g in groups}
    by = {g["N"]: g for g in groups}
    out = []
    for size in sizes:
        g, k = by[size], taken[size]
        taken[size] += 1
        out.append(dict(N=size, Lx=g["Lx"], Ly=g["Ly"], **{f: g[f][k] for f in ("x", "y", "vx", "vy", "rad", "m")}))
    return out


_FIELDS = ("x", "y", "vx", "vy", "rad", "m")


def prepare(case, seed):
    if case["kind"] == "growth":
        systems = []
        for s, n in enumerate(_sizes(case)):
            d = edmd.grow_start(n, case["phi"], 1 + (seed * 7919 + s) % 2000000011)
            d["desc"] = edmd.default_desc(n, d["Lx"], d["Ly"], vr_base=d["vr_base"])
            systems.append(d)
        return dict(case=case, systems=systems)
    systems = _starts(case, seed)
    descs = {}
    for d in systems:
        if d["N"] not in descs:
            descs[d["N"]] = edmd.default_desc(d["N"], d["Lx"], d["Ly"])
        d["desc"] = descs[d["N"]]
    host = {f: np.concatenate([d[f] for d in systems]) for f in _FIELDS}
    state = dict(case=case, engine=edmd.Engine(systems), host=host, seed=seed)
    if case["kind"] == "tangent" and case["systems"] == 1:
        state["vectors"] = _vectors(case, seed)
    return state


def _vectors(case, seed):
    rng = np.random.default_rng([seed, 77])
    q, _ = np.linalg.qr(rng.standard_normal((4 * case["disks"], case["k"])))
    return np.ascontiguousarray(q.T).reshape(case["k"], case["disks"], 4)


def _result(engine, one):
    out = engine.states()
    if one:
        c = engine.counters(0)
        out["ncol"], out["t"] = int(c["ncol"]), float(c["t"])
    else:
        c = engine.all_counters()
        out["ncol"], out["t"] = c["ncol"].astype(np.int64), c["t"]
    return out


def run(state):
    case = state["case"]
    kind = case["kind"]
    one = case["systems"] == 1
    if kind == "growth":
        engine = edmd.Engine(state["systems"])
        engine.advance(flags=edmd.F_STOP_AT_GROW)
        out = _result(engine, one)
        engine.close()
        return out
    engine = state["engine"]
    if kind == "sample":
        engine.sync()
        out = engine.states()
        out["r"], out["g"] = engine.pcf(0, dr=case["dr"], max_r=case["max_r"])
        return out
    engine.load_state(**state["host"])
    if kind == "serial":
        engine.advance(max_coll=case["coll"])
        engine.sync()
        out = _result(engine, one)
        if one:
            out["virial"] = engine.virial(0)
        return out
    if kind == "rounds":
        engine.advance_rounds(t_stop=case["t"], flags=edmd.F_EXACT, radius=3 if case["disks"] <= 20000 else 4)
        engine.sync()
        out = _result(engine, one)
        out["virial"] = engine.virial(0)
        return out
    if kind == "tangent":
        if one:
            vectors, exponents = engine.tangent(case["k"], case["coll"], case["qr"], vectors=state["vectors"])
            return dict(vectors=vectors, exponents=exponents)
        exponents = engine.tangent_batch(case["k"], case["coll"], case["qr"], seed=state["seed"])
        engine.sync()
        return dict(_result(engine, one), exponents=exponents)
    if one:
        msd, g = engine.msd_gradient(case["coll"], ckpt_every=case["ckpt"])
    else:
        msd, g = engine.msd_gradient_batch(case["coll"], ckpt_every=case["ckpt"])
    return dict(g, msd=msd)


# ------------------------------------------------------------------ work

def _collisions(case):
    """Collisions of one pass, all systems (an estimate where a time bounds the run)."""
    if "coll" in case:
        return case["coll"] * case["systems"]
    disks = sum(_sizes(case))
    if case["kind"] == "growth":
        return 12 * disks
    return 4.2 * disks * case["t"]


def work(case):
    disks = sum(_sizes(case))
    move = 2 * 48 * disks                            # state in and out
    if case["kind"] == "sample":
        pairs = disks * case["phi"] * case["max_r"] ** 2 / 2
        return {"bytes": 2 * 48 * disks, "flops": 10 * pairs}
    n = _collisions(case)
    # per collision: 2.6 predictions over 19.4 candidate pairs, 48 bytes each, and the events and disks written
    b, f = n * 1300.0, n * 19.4 * 25
    if case["kind"] == "tangent":
        rows = 4 * disks * case["k"]
        qrs = -(-case["coll"] // case["qr"]) + 1
        b += 2 * 8 * rows + n * 2 * 2 * 4 * case["k"] * 8 + qrs * 2 * 8 * rows
        f += n * 70 * case["k"] + qrs * 4 * rows * case["k"]
    if case["kind"] == "gradient":
        b, f = 2 * b, 2 * f + n * 100
    return {"bytes": b + move, "flops": f}


# ------------------------------------------------------------------ the same in plain Python, 64 bits

class _Box:
    """Event-driven dynamics of one system, events in time order from a heap."""

    def __init__(self, d, dtime=100.0):
        self.N, self.Lx, self.Ly = d["N"], d["Lx"], d["Ly"]
        self.x, self.y, self.vx, self.vy, self.rad, self.m = (list(map(float, d[f])) for f in _FIELDS)
        self.nx, self.ny = int(self.Lx / 2), int(self.Ly / 2)
        self.sx, self.sy = self.Lx / self.nx, self.Ly / self.ny
        self.tl = [0.0] * self.N
        self.hits = [0] * self.N
        self.cx = [min(int(v / self.sx), self.nx - 1) for v in self.x]
        self.cy = [min(int(v / self.sy), self.ny - 1) for v in self.y]
        self.cells = [[] for _ in range(self.nx * self.ny)]
        for i in range(self.N):
            self.cells[self.cy[i] * self.nx + self.cx[i]].append(i)
        self.t, self.ncol, self.virial, self.log = 0.0, 0, [0.0] * 4, []
        self.heap, self.order = [], 0
        self.now = [[0, 0] for _ in range(self.N)]   # newest crossing and collision event of each disk
        self.dtime = dtime
        heapq.heappush(self.heap, (1.0, -1, -1, 2, 0, 0))
        for i in range(self.N):
            self.next_wall(i)
            self.next_hit(i)

    def push(self, t, i, what, j, stamp):
        self.order += 1
        self.now[i][what] = self.order
        heapq.heappush(self.heap, (t, self.order, i, what, j, stamp))

    def fly(self, i, t):
        dt = t - self.tl[i]
        self.tl[i] = t
        self.x[i] = (self.x[i] + dt * self.vx[i]) % self.Lx
        self.y[i] = (self.y[i] + dt * self.vy[i]) % self.Ly

    def near(self, d, length):
        return d - length if d >= length / 2 else d + length if d < -length / 2 else d

    def next_wall(self, i):
        best, way = math.inf, 0
        for v, p, c, s, length, k in ((self.vx[i], self.x[i], self.cx[i], self.sx, self.Lx, 0), (self.vy[i], self.y[i], self.cy[i], self.sy, self.Ly, 2)):
            if v == 0:
                continue
            dt = self.near((c + (v > 0)) * s - p, length) / v
            if dt < best:
                best, way = dt, k + (v > 0)
        self.push(self.t + best, i, 0, way, 0)

    def next_hit(self, i):
        t, x, y, vx, vy, r = self.t, self.x[i], self.y[i], self.vx[i], self.vy[i], self.rad[i]
        best, who = math.inf, -1
        for oy in (-1, 0, 1):
            row = (self.cy[i] + oy) % self.ny * self.nx
            for ox in (-1, 0, 1):
                for j in self.cells[row + (self.cx[i] + ox) % self.nx]:
                    if j == i:
                        continue
                    late = t - self.tl[j]
                    ux, uy = self.vx[j] - vx, self.vy[j] - vy
                    dx = self.near(self.x[j] + late * self.vx[j] - x, self.Lx)
                    dy = self.near(self.y[j] + late * self.vy[j] - y, self.Ly)
                    b = dx * ux + dy * uy
                    if b > 0:
                        continue
                    v2 = ux * ux + uy * uy
                    det = b * b - v2 * (dx * dx + dy * dy - 4 * r * self.rad[j])
                    if det >= 0 and (-b - math.sqrt(det)) / v2 < best:
                        best, who = (-b - math.sqrt(det)) / v2, j
        if who >= 0:
            self.push(t + best, i, 1, who, self.hits[who])
        else:
            self.order += 1
            self.now[i][1] = self.order

    def collide(self, i, j):
        self.fly(j, self.t)
        self.ncol += 1
        self.hits[i] += 1
        self.hits[j] += 1
        dx, dy = self.near(self.x[j] - self.x[i], self.Lx), self.near(self.y[j] - self.y[i], self.Ly)
        ux, uy = self.vx[j] - self.vx[i], self.vy[j] - self.vy[i]
        mi, mj = self.m[i], self.m[j]
        f = 2 / (mi + mj) * (dx * ux + dy * uy) / (4 * self.rad[i] * self.rad[j])
        self.log.append((i, j, self.t, dx, dy, ux, uy, f))
        for k, (p, q) in enumerate(((dx, dx), (dy, dy), (dx, dy), (dy, dx))):
            self.virial[k] += mi * mj * f * p * q
        self.vx[i] += f * mj * dx
        self.vy[i] += f * mj * dy
        self.vx[j] -= f * mi * dx
        self.vy[j] -= f * mi * dy

    def run(self, coll=math.inf, t_stop=math.inf):
        while self.ncol < coll:
            t, order, i, what, j, stamp = self.heap[0]
            if what < 2 and self.now[i][what] != order:
                heapq.heappop(self.heap)
                continue
            if t >= t_stop:
                break
            heapq.heappop(self.heap)
            self.t = t
            if what == 2:
                for k in range(self.N):
                    self.fly(k, t)
                heapq.heappush(self.heap, (t + self.dtime, -1, -1, 2, 0, 0))
                continue
            self.fly(i, t)
            if what == 0:
                self.cells[self.cy[i] * self.nx + self.cx[i]].remove(i)
                if j < 2:
                    self.cx[i] = (self.cx[i] + 2 * j - 1) % self.nx
                else:
                    self.cy[i] = (self.cy[i] + 2 * (j - 2) - 1) % self.ny
                self.cells[self.cy[i] * self.nx + self.cx[i]].append(i)
                self.next_wall(i)
            elif stamp == self.hits[j]:
                self.collide(i, j)
                for k in (i, j):
                    self.next_wall(k)
                self.next_hit(i)
                self.next_hit(j)
                continue
            self.next_hit(i)

    def states(self):
        for i in range(self.N):
            self.fly(i, self.t)
        return dict(x=self.x, y=self.y, vx=self.vx, vy=self.vy, rad=self.rad, m=self.m)


def _tangent(box, log, R, clock):
    """The tangent map over collisions; R is [4 N][K], every disk's rows at its own time `clock`."""
    for i, j, t, dx, dy, ux, uy, f in log:
        xi, yi, vxi, vyi = R[4 * i], R[4 * i + 1], R[4 * i + 2], R[4 * i + 3]
        xj, yj, vxj, vyj = R[4 * j], R[4 * j + 1], R[4 * j + 2], R[4 * j + 3]
        ai, aj = t - clock[i], t - clock[j]
        xi, yi, xj, yj = xi + vxi * ai, yi + vyi * ai, xj + vxj * aj, yj + vyj * aj
        mi, mj = box.m[i], box.m[j]
        rv = dx * ux + dy * uy
        ex, ey, wx, wy = xj - xi, yj - yi, vxj - vxi, vyj - vyi
        tc = -(dx * ex + dy * ey) / rv
        cx, cy = ex + ux * tc, ey + uy * tc
        df = f / rv * (ux * cx + uy * cy + dx * wx + dy * wy)
        px, py = df * dx + f * cx, df * dy + f * cy
        R[4 * i], R[4 * i + 1] = xi - f * mj * dx * tc, yi - f * mj * dy * tc
        R[4 * j], R[4 * j + 1] = xj + f * mi * dx * tc, yj + f * mi * dy * tc
        R[4 * i + 2], R[4 * i + 3] = vxi + mj * px, vyi + mj * py
        R[4 * j + 2], R[4 * j + 3] = vxj - mi * px, vyj - mi * py
        clock[i] = clock[j] = t


def _gradient(box, log, x0, y0):
    """Final mean-square displacement and its gradient, the transposed maps backwards over the log."""
    N, T = box.N, box.t
    late = T - np.array(box.tl)
    # positions at T, unwrapped displacements by the nearest image
    ux = np.array(box.x) + np.array(box.vx) * late - x0
    uy = np.array(box.y) + np.array(box.vy) * late - y0
    ux -= box.Lx * np.rint(ux / box.Lx)
    uy -= box.Ly * np.rint(uy / box.Ly)
    ux -= ux.mean()
    uy -= uy.mean()
    msd = float((ux * ux + uy * uy).sum() / N)
    A = np.zeros((N, 4))
    A[:, 0], A[:, 1] = 2 * ux / N, 2 * uy / N
    A = [list(map(float, a)) for a in A]
    clock = [T] * N
    for i, j, t, dx, dy, vx, vy, f in reversed(log):
        mi, mj = box.m[i], box.m[j]
        a, b = A[i], A[j]
        gxi, gyi, gxj, gyj = a[0], a[1], b[0], b[1]
        gvxi, gvyi = a[2] + gxi * (clock[i] - t), a[3] + gyi * (clock[i] - t)
        gvxj, gvyj = b[2] + gxj * (clock[j] - t), b[3] + gyj * (clock[j] - t)
        rv = dx * vx + dy * vy
        px, py = mj * gvxi - mi * gvxj, mj * gvyi - mi * gvyj
        gt = -f * mj * (dx * gxi + dy * gyi) + f * mi * (dx * gxj + dy * gyj)
        s = f / rv * (dx * px + dy * py)
        cx, cy = f * px + s * vx, f * py + s * vy
        gt += vx * cx + vy * cy
        rx, ry = cx - gt / rv * dx, cy - gt / rv * dy
        A[i] = [gxi - rx, gyi - ry, gvxi - s * dx, gvyi - s * dy]
        A[j] = [gxj + rx, gyj + ry, gvxj + s * dx, gvyj + s * dy]
        clock[i] = clock[j] = t
    A, clock = np.array(A), np.array(clock)
    A[:, 2] += A[:, 0] * clock
    A[:, 3] += A[:, 1] * clock
    return msd, dict(vx=A[:, 2], vy=A[:, 3], x=A[:, 0] - 2 * ux / N, y=A[:, 1] - 2 * uy / N)


def _pair_counts(d, dr, max_r):
    nb = int(max_r / dr)
    counts = np.zeros(nb, np.int64)
    order = np.argsort(d["x"], kind="stable")
    x, y, N = d["x"][order], d["y"][order], d["N"]
    xx = np.concatenate([x, x + d["Lx"]])
    yy = np.concatenate([y, y])
    end = np.searchsorted(xx, x + max_r, side="right")
    step = 256
    for a in range(0, N, step):
        b = min(N, a + step)
        cols = np.arange(a + 1, end[b - 1])
        dx = xx[cols][None, :] - x[a:b, None]
        dy = yy[cols][None, :] - y[a:b, None]
        dy -= d["Ly"] * (dy >= d["Ly"] / 2)
        dy += d["Ly"] * (dy < -d["Ly"] / 2)
        rows = np.arange(a, b)
        own = (cols[None, :] > rows[:, None]) & (cols[None, :] < end[rows][:, None]) & (np.abs(dy) < max_r)
        r = np.sqrt(dx[own] ** 2 + dy[own] ** 2)
        r = r[r < max_r]
        k = (r / dr).astype(np.int64)
        counts += np.bincount(k[k < nb], minlength=nb)[:nb]
    return counts


def exact(case, seed):
    kind = case["kind"]
    if kind == "growth":
        return None
    disks = sum(_sizes(case))
    if kind == "sample":
        if disks > 120000:
            return None
        d = _starts(case, seed)[0]
        counts = _pair_counts(d, case["dr"], case["max_r"])
        r = (np.arange(len(counts)) + 0.5) * case["dr"]
        g = 2.0 * counts / (2 * math.pi * r * case["dr"] * (d["N"] / (d["Lx"] * d["Ly"])) * d["N"])
        return dict({f: d[f] for f in _FIELDS}, r=r, g=g)
    if disks + 4 * _collisions(case) > 1500000 or (kind == "tangent" and case["systems"] > 1):
        return None
    starts = _starts(case, seed)
    if kind == "tangent":
        box = _Box(starts[0])
        R = np.ascontiguousarray(_vectors(case, seed).reshape(case["k"], -1).T)
        clock = [0.0] * box.N
        logs = np.zeros(case["k"])
        done = 0
        while done < case["coll"]:
            want = min(case["qr"], case["coll"] - done)
            box.log = []
            box.run(coll=done + want)
            _tangent(box, box.log, R, clock)
            late = np.repeat(box.t - np.array(clock), 4) * np.tile([1.0, 1.0, 0.0, 0.0], box.N)
            R += late[:, None] * R[np.arange(4 * box.N) + np.tile([2, 2, 0, 0], box.N)]
            clock = [box.t] * box.N
            Q, U = np.linalg.qr(R)
            sign = np.sign(np.diag(U))
            R = Q * sign
            logs += np.log(np.abs(np.diag(U)))
            done += want
        return dict(vectors=np.ascontiguousarray(R.T).reshape(case["k"], box.N, 4), exponents=logs / box.t)
    if kind == "gradient":
        parts = []
        for d in starts:
            box = _Box(d)
            box.run(coll=case["coll"])
            parts.append(_gradient(box, box.log, d["x"], d["y"]))
        g = {f: np.concatenate([p[1][f] for p in parts]) for f in ("vx", "vy", "x", "y")}
        msd = parts[0][0] if case["systems"] == 1 else np.array([p[0] for p in parts])
        return dict(g, msd=msd)
    boxes = [_Box(d) for d in starts]
    for box in boxes:
        box.run(coll=case["coll"]) if kind == "serial" else box.run(t_stop=case["t"])
    got = [b.states() for b in boxes]
    out = {f: np.concatenate([np.asarray(s[f]) for s in got]) for f in _FIELDS}
    if case["systems"] == 1:
        out.update(ncol=boxes[0].ncol, t=boxes[0].t, virial=np.array(boxes[0].virial))
    else:
        out.update(ncol=np.array([b.ncol for b in boxes]), t=np.array([b.t for b in boxes]))
    return out
