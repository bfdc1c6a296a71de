"""Performance cases: what programs built on this package ask of it.

Each case is one call, or the few calls a driver makes per batch, through the
public entry points of ``mipt_gb300``. ``kind`` names the family:

layer   one layer of a single trajectory on ``Engine``: a brickwork layer of
        two-qubit gates, then the joint Born measurement of some sites.
entropy S_vN (``entropy_svd``) or S_2 (``renyi2``) of one subsystem.
rho3    the three-site density matrices of the ring triples.
batch   ``Batch.run``: host draw, upload, every layer, observables, fetch.
free    the free-energy protocol: random product initial states, workspace
        draw, all layers, half-chain S_vN at the observation steps.
ff      monitored free fermions (``ff_run``).
gmn     genuine multipartite negativity of three-qubit states.

An FP32 run's results carry FP32 accuracy, whatever the width of the array
they are handed over in; they are returned as float32, the type of the states
they were computed from, and the results of FP64 runs as float64.
"""
import math

import numpy as np
import torch

import mipt_gb300 as mg

MASK64 = (1 << 64) - 1
# A full check in 64 bits has to end within about 20 seconds: amplitude-layers
# evolved, FP64 multiply-adds of Gram matrices, rows^3 of eigenvalue problems.
EVOLVE_LIMIT = 1 << 32
GRAM_LIMIT = 3e12
EIG_LIMIT = 2.5e10


# ------------------------------------------------------------------- cases
def listed():
    return [
        # One layer of the smallest chains a driver steps through by itself:
        # launch and synchronisation latency, no bandwidth.
        dict(name="layer n10 f64", kind="layer", n=10, fp64=True, odd=False, closed=False, p=0.2),
        # The same step of a large single trajectory (a closed ring's odd layer).
        dict(name="layer n26 f32", kind="layer", n=26, fp64=False, odd=True, closed=True, p=0.15),
        # The half cut of sim_tmi / entropy on a 16-qubit FP64 state: Gram and
        # 256-row FP64 spectrum of one matrix.
        dict(name="svn n16 k8 f64", kind="entropy", n=16, fp64=True, order=1, k=8, start=3, step=1),
        # Renyi-2 of an interleaved subsystem of a large FP32 state (odd n,
        # gathered rows).
        dict(name="renyi2 n23 k11 f32", kind="entropy", n=23, fp64=False, order=2, k=11, start=0, step=2),
        # mipt.exe's final observable: rho3 of every ring triple.
        dict(name="rho3 n20 f32", kind="rho3", n=20, fp64=False),
        # The plain FP64 method: L = 12 open chain, 200 trajectories, every
        # observable after every layer.
        dict(name="batch L12 f64 all observables", kind="batch", n=12, periods=12, count=200, fp64=True,
             closed=False, circuit=1, lattice_x=0, svn=True, s2=True, tmi_vn=True, tmi_s2=True, every=1,
             region=0, rho3=False, p_lo=0.2, p_hi=0.2),
        # The headline workload: 32 trajectories of the L = 24 ring, 48
        # layers, final half-chain S_2.
        dict(name="batch L24 f32 final S2", kind="batch", n=24, periods=24, count=32, fp64=False,
             closed=True, circuit=1, lattice_x=0, svn=False, s2=True, tmi_vn=False, tmi_s2=False, every=0,
             region=0, rho3=False, p_lo=0.05, p_hi=0.35),
        # One length of the mixed-length scan: per-layer half-chain S_2 and
        # TMI of the quarters.
        dict(name="batch L20 f32 per-layer S2 TMI", kind="batch", n=20, periods=10, count=48, fp64=False,
             closed=True, circuit=1, lattice_x=0, svn=False, s2=True, tmi_vn=False, tmi_s2=True, every=1,
             region=0, rho3=False, p_lo=0.05, p_hi=0.35),
        # The 4 x 7 lattice (2 GiB state): half-system S_2, S_vN of two rows
        # and the lattice triples' rho3, one four-colour cycle.
        dict(name="lattice 4x7 f32 observed", kind="batch", n=28, periods=2, count=1, fp64=False,
             closed=True, circuit=1, lattice_x=4, svn=False, s2=True, tmi_vn=False, tmi_s2=False, every=1,
             region=8, rho3=True, p_lo=0.15, p_hi=0.15),
        # The free-energy protocol's batch, FP32 states, S_vN early on.
        dict(name="free energy N16 f32", kind="free", n=16, layers=64, count=64, fp64=False, p=0.1, points=17),
        # Free fermions, the plain FP64 method at the configuration's size.
        dict(name="free fermions N128 f64", kind="ff", n=128, depth=32, count=304, fp64=True, p=0.2, closed=True,
             every=16),
        # rho3 -> GMN: cold start to a certified gap of 1e-6.
        dict(name="gmn 2048", kind="gmn", count=2048, max_iter=600, fp64=False),
    ]


def draw(rng):
    """One more case of the same ranges."""
    kind = rng.choice(["layer", "layer", "entropy", "entropy", "rho3", "batch", "batch", "batch", "free", "ff", "gmn"])
    fp64 = rng.random() < 0.4
    if kind == "layer":
        return dict(kind=kind, n=rng.randint(5, 13) * 2 - rng.randint(0, 1), fp64=fp64, odd=rng.random() < 0.5,
                    closed=rng.random() < 0.5, p=round(rng.uniform(0.05, 0.4), 3))
    if kind == "entropy":
        order = rng.choice([1, 2])
        n = rng.randint(10, 17 if order == 1 else 23)
        k = rng.randint(3, min(9 if order == 1 else 11, n // 2))
        step = rng.choice([1, 1, 2]) if 2 * k <= n else 1
        return dict(kind=kind, n=n, fp64=fp64 and n <= 20, order=order, k=k,
                    start=rng.randint(0, n - 1 - step * (k - 1)), step=step)
    if kind == "rho3":
        return dict(kind=kind, n=rng.randint(8, 23), fp64=fp64)
    if kind == "batch":
        shape = rng.choice(["small", "small", "large", "rppu", "lattice"])
        c = dict(kind=kind, circuit=1, lattice_x=0, closed=rng.random() < 0.7, fp64=fp64, svn=False, s2=True,
                 tmi_vn=False, tmi_s2=False, every=0, region=0, rho3=False, p_lo=round(rng.uniform(0.03, 0.2), 3),
                 p_hi=round(rng.uniform(0.2, 0.45), 3))
        if shape == "small":
            n = rng.choice([8, 10, 12, 14, 16])
            c.update(n=n, periods=rng.randint(3, n), count=int(2 ** rng.uniform(1, 20 - n) + rng.randint(1, 30)),
                     svn=n <= 14 and rng.random() < 0.6, tmi_vn=n in (8, 12), tmi_s2=n % 4 == 0, every=rng.choice([1, 2]),
                     rho3=rng.random() < 0.4)
        elif shape == "large":
            n = rng.choice([18, 20, 22, 24])
            c.update(n=n, periods=rng.randint(3, 12), count=rng.randint(1, 1 << min(6, 27 - n)),
                     fp64=fp64 and n <= 20, every=rng.choice([0, 0, 1]), tmi_s2=n == 20 and rng.random() < 0.4)
        elif shape == "rppu":
            n = rng.choice([10, 14, 18, 22])
            c.update(n=n, periods=rng.randint(3, 10), count=rng.randint(2, 33), closed=True,
                     circuit=rng.choice([2, 4]), fp64=fp64 and n <= 18)
        else:
            x, y = rng.choice([(3, 4), (4, 4), (4, 5), (4, 6), (6, 4)])
            c.update(n=x * y, lattice_x=x, periods=2 * rng.randint(1, 3), count=rng.randint(1, 6), closed=True,
                     fp64=fp64 and x * y <= 16, every=1, region=rng.randint(3, 7), rho3=rng.random() < 0.5)
        return c
    if kind == "free":
        n = rng.choice([8, 10, 12, 14, 16])
        return dict(kind=kind, n=n, layers=2 * rng.randint(2 * n, 4 * n), count=rng.randint(20, 80), fp64=fp64,
                    p=round(rng.uniform(0.05, 0.3), 3), points=rng.randint(5, n + 1))
    if kind == "ff":
        n = rng.choice([16, 24, 48, 64, 96, 128])
        return dict(kind=kind, n=n, depth=rng.randint(8, 32), count=rng.randint(10, 300), fp64=rng.random() < 0.7,
                    p=round(rng.uniform(0.1, 0.3), 3), closed=rng.random() < 0.7, every=rng.choice([0, 8, 16]))
    fp64 = rng.random() < 0.2
    return dict(kind="gmn", count=int(2 ** rng.uniform(4, 8 if fp64 else 11)) + rng.randint(0, 7),
                max_iter=100 if fp64 else rng.choice([200, 400, 600]), fp64=fp64)


# ----------------------------------------------------- inputs, 64-bit tools
def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _apply(psi, n, a, b, u):
    """Two-qubit gate u (index bit 0 = qubit a) on psi[..., 2^n]."""
    lead = psi.shape[:-1]
    m = len(lead)
    t = psi.reshape(lead + (2,) * n)
    ax = (m + n - 1 - b, m + n - 1 - a)
    t = torch.movedim(t, ax, (0, 1)).reshape(4, -1)
    t = torch.as_tensor(u, dtype=psi.dtype, device=psi.device).reshape(4, 4) @ t
    t = t.reshape((2, 2) + lead + (2,) * (n - 2))
    return torch.movedim(t, (0, 1), ax).reshape(lead + (-1,))


def _haar_gates(rng, count):
    z = rng.normal(size=(count, 4, 4)) + 1j * rng.normal(size=(count, 4, 4))
    q, r = np.linalg.qr(z)
    d = np.diagonal(r, axis1=1, axis2=2)
    return q * (d / abs(d))[:, None, :]


def _bonds(n, odd, closed):
    stop = n if (closed and odd and n > 2 and n % 2 == 0) else n - 1
    return [(i, (i + 1) % n) for i in range(1 if odd else 0, stop, 2)]


def _trajectory_state(n, seed, fp64):
    """A state as a monitored circuit leaves it: a few brickwork layers with
    projective measurements between them, then normalised."""
    rng = np.random.default_rng([seed, n, 77])
    psi = torch.zeros(1 << n, dtype=torch.complex128 if fp64 else torch.complex64, device=_device())
    psi[0] = 1
    for t in range(6):
        for (a, b), u in zip(_bonds(n, t % 2 == 1, True), _haar_gates(rng, n // 2 + 1)):
            psi = _apply(psi, n, a, b, u)
        if t in (2, 4):
            for q in np.nonzero(rng.random(n) < 0.12)[0]:
                v = psi.reshape(-1, 2, 1 << int(q))
                w = torch.linalg.vector_norm(v, dim=(0, 2))
                v[:, int(w[0] >= w[1])] = 0
                psi = v.reshape(-1)
            psi = psi / torch.linalg.vector_norm(psi)
    return (psi / torch.linalg.vector_norm(psi)).contiguous()


def _rows(psi, n, kept):
    """psi[..., 2^n] as [..., 2^k, 2^(n-k)], row bit i = qubit kept[i]."""
    lead = psi.shape[:-1]
    m = len(lead)
    t = psi.reshape(lead + (2,) * n)
    rest = [q for q in range(n) if q not in kept]
    order = list(range(m)) + [m + n - 1 - q for q in reversed(kept)] + [m + n - 1 - q for q in reversed(rest)]
    return t.permute(order).reshape(lead + (1 << len(kept), 1 << len(rest)))


def _gram_work(n, k):
    small, large = 1 << min(k, n - k), 1 << max(k, n - k)
    return 4.0 * small * small * large


def _entropy(psi, n, kept, order):
    """Entropy in bits of `kept` for psi[..., 2^n] in 64 bits."""
    m = _rows(psi, n, kept)
    if m.shape[-2] > m.shape[-1]:
        m = m.transpose(-1, -2)
    rho = m @ m.transpose(-1, -2).conj()
    if order == 2:
        pur = (rho.real ** 2 + rho.imag ** 2).sum((-1, -2))
        return torch.where(pur >= 1, torch.zeros_like(pur), -torch.log2(pur))
    lam = torch.linalg.eigvalsh(rho)
    s = torch.where(lam > 1e-15, -lam * torch.log2(lam.clamp_min(1e-300)), torch.zeros_like(lam)).sum(-1)
    return torch.where(s.abs() < 1e-12, torch.zeros_like(s), s)


def _measure(psi, n, sites, u):
    """Joint Born measurement of ascending sites with one uniform: the
    outcomes' bits, log P, the collapsed state."""
    w = _rows(psi, n, sites)
    w = (w.real ** 2 + w.imag ** 2).sum(-1).cpu().numpy()
    c = np.cumsum(w)
    at = min(int(np.searchsorted(c, u * c[-1], side="right")), len(w) - 1)
    bits = [(at >> i) & 1 for i in range(len(sites))]
    for q, o in zip(sites, bits):
        psi = psi.reshape(-1, 2, 1 << q).clone()
        psi[:, 1 - o] = 0
        psi = psi.reshape(-1)
    return bits, math.log(w[at] / c[-1]), psi / math.sqrt(w[at])


# The seed streams of a trajectory (std::mt19937 as libstdc++ seeds and reads it).
def _splitmix64(v):
    v = (v + 0x9E3779B97F4A7C15) & MASK64
    v = ((v ^ (v >> 30)) * 0xBF58476D1CE4E5B9) & MASK64
    v = ((v ^ (v >> 27)) * 0x94D049BB133111EB) & MASK64
    return v ^ (v >> 31)


def _seed_seq(words, n=624):
    """std::seed_seq::generate."""
    m32 = 0xFFFFFFFF
    s, b = len(words), [0x8B8B8B8B] * n
    t = 11 if n >= 623 else 7
    p = (n - t) // 2
    q = p + t
    mix = lambda x: x ^ (x >> 27)  # noqa: E731
    m = max(s + 1, n)
    for k in range(m):
        r1 = (1664525 * mix(b[k % n] ^ b[(k + p) % n] ^ b[(k - 1) % n])) & m32
        r2 = (r1 + (s if k == 0 else k % n + words[k - 1] if k <= s else k % n)) & m32
        b[(k + p) % n] = (b[(k + p) % n] + r1) & m32
        b[(k + q) % n] = (b[(k + q) % n] + r2) & m32
        b[k % n] = r2
    for k in range(m, m + n):
        r3 = (1566083941 * mix((b[k % n] + b[(k + p) % n] + b[(k - 1) % n]) & m32)) & m32
        r4 = (r3 - k % n) & m32
        b[(k + p) % n] ^= r3
        b[(k + q) % n] ^= r4
        b[k % n] = r4
    return b


class _Stream:
    """Uniform doubles of an std::mt19937, two words each."""

    def __init__(self, seed, workspace=False):
        if workspace:
            self.bits = np.random.RandomState(seed)._bit_generator
        else:
            self.bits = np.random.MT19937()
            self.bits.state = {"bit_generator": "MT19937", "state": {
                "key": np.array(_seed_seq([seed & 0xFFFFFFFF, seed >> 32]), np.uint32), "pos": 624}}
        self.have = np.zeros(0)

    def take(self, k):
        if len(self.have) < k:
            w = self.bits.random_raw(2 * max(k, 8192)).astype(np.float64).reshape(-1, 2)
            self.have = np.concatenate([self.have, (w[:, 0] + w[:, 1] * 4294967296.0) / 18446744073709551616.0])
        out, self.have = self.have[:k], self.have[k:]
        return out

    def normals(self, k):
        """k (even) normals of std::normal_distribution (polar method)."""
        out = np.zeros(0)
        while len(out) < k:
            need = (k - len(out)) // 2
            v = 2.0 * self.take(2 * need).reshape(-1, 2) - 1.0
            r2 = (v ** 2).sum(1)
            v, r2 = v[(r2 <= 1) & (r2 > 0)], r2[(r2 <= 1) & (r2 > 0)]
            out = np.concatenate([out, (v[:, ::-1] * np.sqrt(-2.0 * np.log(r2) / r2)[:, None]).reshape(-1)])
        return out


def _gram_schmidt(z):
    """Columns of z[g, r, c], orthonormalised left to right."""
    q = np.zeros_like(z)
    for c in range(z.shape[2]):
        v = z[:, :, c].copy()
        for k in range(c):
            v -= q[:, :, k] * (q[:, :, k].conj() * v).sum(1)[:, None]
        q[:, :, c] = v / np.sqrt((abs(v) ** 2).sum(1))[:, None]
    return q


def _lattice_bonds(x, y, colour):
    """Bonds of one colour of the x by y lattice (site = row * x + column)."""
    horizontal = colour < 2
    out = []
    for line in range(y if horizontal else x):
        length = x if horizontal else y
        site = [line * x + i if horizontal else i * x + line for i in range(length)]
        if line % 2 == colour % 2:
            out += [(site[i], site[i + 1]) for i in range(0, length - 1, 2)]
        else:
            if length % 2 == 0:
                out.append((site[0], site[-1]))
            out += [(site[i], site[i + 1]) for i in range(1, length - 1, 2)]
    return out


def _haar_record(seed, n, layers, p, closed, lattice_x=0, workspace=False):
    """The random record of a Haar trajectory: per layer its bonds, unitaries,
    measured sites and measurement uniforms (chunks of 16 sites)."""
    gates = _Stream(seed, workspace)
    meas = _Stream(seed ^ 0x9E3779B9, True) if workspace else _Stream(_splitmix64(seed ^ 0xA0761D0D))
    out = []
    for t in range(layers):
        bonds = _lattice_bonds(lattice_x, n // lattice_x, t % 4) if lattice_x else _bonds(n, t % 2 == 1, closed)
        z = gates.normals(32 * len(bonds)).reshape(-1, 4, 4, 2)  # gate, column, row, (im, re)
        u = _gram_schmidt(np.swapaxes(z[..., 1] + 1j * z[..., 0], 1, 2))
        sites = [int(s) for s in np.nonzero(gates.take(n) < p)[0]] if p > 0 else []
        out.append((bonds, u, sites, meas.take((len(sites) + 15) // 16)))
    return out


class _Mt64:
    """std::mt19937_64's uniform doubles."""

    def __init__(self, seed):
        self.s = [seed & MASK64]
        for i in range(1, 312):
            self.s.append((6364136223846793005 * (self.s[-1] ^ (self.s[-1] >> 62)) + i) & MASK64)
        self.at = 312

    def uniform(self):
        s = self.s
        if self.at == 312:
            for i in range(312):
                v = (s[i] & 0xFFFFFFFF80000000) | (s[(i + 1) % 312] & 0x7FFFFFFF)
                s[i] = s[(i + 156) % 312] ^ (v >> 1) ^ (0xB5026F5AA96619E9 if v & 1 else 0)
            self.at = 0
        v = s[self.at]
        self.at += 1
        v ^= (v >> 29) & 0x5555555555555555
        v ^= (v << 17) & 0x71D67FFFEDA60000
        v ^= (v << 37) & 0xFFF7EEE000000000
        v ^= v >> 43
        return min(float(v) / 18446744073709551616.0, math.nextafter(1.0, 0.0))


def _product_state(seed, n, fp64):
    """The free-energy protocol's random product state, rounded where it is stored."""
    rng, real = _Mt64(seed), np.complex128 if fp64 else np.complex64
    out = np.ones(1, real)
    for _ in range(n):
        theta = math.acos(min(1.0, max(-1.0, 1.0 - 2.0 * rng.uniform())))
        phi = 2.0 * math.pi * rng.uniform()
        site = [math.cos(0.5 * theta), math.sin(0.5 * theta) * complex(math.cos(phi), math.sin(phi))]
        out = np.concatenate([(out.astype(np.complex128) * f).astype(real) for f in site])
    return out


def _layer(psi, n, layer):
    """One recorded layer on psi[2^n]: outcome mask, surprisal, state."""
    bonds, u, sites, uniforms = layer
    for (a, b), g in zip(bonds, u):
        psi = _apply(psi, n, a, b, g)
    mask, logp = 0, 0.0
    for c, x in enumerate(uniforms):
        chunk = sites[16 * c: 16 * c + 16]
        bits, lp, psi = _measure(psi, n, chunk, x)
        logp += lp
        mask |= sum(o << q for q, o in zip(chunk, bits))
    return mask, -logp, psi


# ------------------------------------------------------- prepare, run, work
def _real(x, fp64):
    return np.asarray(x, np.float64 if fp64 else np.float32)


def _kept(case):
    return [case["start"] + case["step"] * i for i in range(case["k"])]


def _ring(n):
    return [[i, (i + 1) % n, (i + 2) % n] for i in range(n)]


def _layer_inputs(case, seed):
    n = case["n"]
    rng = np.random.default_rng([seed, 5])
    bonds = _bonds(n, case["odd"], case["closed"])
    gates = _haar_gates(rng, len(bonds))
    sites = sorted(int(q) for q in rng.choice(n, size=max(1, round(case["p"] * n)), replace=False))
    return _trajectory_state(n, seed, case["fp64"]), bonds, gates, sites, rng.random((len(sites) + 15) // 16)


def _seeds(seed, count, bits=64):
    return [_splitmix64((seed * 1000003 + i) & MASK64) & ((1 << bits) - 1) for i in range(count)]


def _p_of(case):
    return np.array([case["p_lo"] + (case["p_hi"] - case["p_lo"]) * (i % 16) / 15.0 for i in range(case["count"])])


def _three_qubit_states(case, seed):
    """Half mixtures of GHZ, W and product states with white noise, half
    three-site states of random pure five-qubit states, as rho3 files hold them."""
    rng = np.random.default_rng([seed, 9])
    count = case["count"]
    ghz, w = np.zeros(8, complex), np.zeros(8, complex)
    ghz[[0, 7]], w[[1, 2, 4]] = 2 ** -0.5, 3 ** -0.5
    weights = rng.dirichlet(np.ones(3), size=count)
    noise = rng.random(count)
    prod = rng.normal(size=(count, 3, 2)) + 1j * rng.normal(size=(count, 3, 2))
    prod /= np.linalg.norm(prod, axis=2, keepdims=True)
    prod = np.einsum("na,nb,nc->nabc", prod[:, 0], prod[:, 1], prod[:, 2]).reshape(count, 8)
    rho = (weights[:, 0, None, None] * np.outer(ghz, ghz.conj()) + weights[:, 1, None, None] * np.outer(w, w.conj())
           + weights[:, 2, None, None] * prod[:, :, None] * prod[:, None, :].conj())
    rho = (1 - noise)[:, None, None] * rho + noise[:, None, None] * np.eye(8) / 8
    psi = rng.normal(size=(count, 8, 4)) + 1j * rng.normal(size=(count, 8, 4))
    psi /= np.linalg.norm(psi, axis=(1, 2), keepdims=True)
    rho[::2] = np.einsum("nik,njk->nij", psi, psi.conj())[::2]
    return rho


def _blocks(n):
    return [1, n // 8, n // 4, n // 2, n - 1]


def _make_batch(case):
    obs = (mg.OBS_SVN_HALF * case["svn"] | mg.OBS_S2_HALF * case["s2"] | mg.OBS_TMI_VN * case["tmi_vn"]
           | mg.OBS_TMI_S2 * case["tmi_s2"])
    x = case["lattice_x"]
    b = mg.Batch(case["n"], case["periods"], case["count"], closed=case["closed"], fp64=case["fp64"],
                 observables=obs, observe_every=case["every"], rho3=case["rho3"], circuit=case["circuit"],
                 fermion_trace=case["circuit"] == 2, lattice=(x, case["n"] // x) if x else None)
    if case["region"]:
        b.add_region(list(range(case["region"])), 1)
    if case["rho3"]:
        b.set_rho3_subsystems(_triples(case))
    return b


def _triples(case):
    return [[0, 1, 2], [0, case["lattice_x"] or 3, case["n"] - 1], [case["n"] // 2, 1, 2]]


class _Array:
    """A device buffer for torch.as_tensor; the tensor keeps this object, and it the buffer's owner."""

    def __init__(self, owner, pointer, shape, fp64):
        self.owner = owner
        self.__cuda_array_interface__ = dict(data=(pointer, False), shape=shape, typestr="<c16" if fp64 else "<c8",
                                             version=3, strides=None)


def _batch_states(batch, case):
    return torch.as_tensor(_Array(batch, batch.state_ptr(0), (case["count"], 1 << case["n"]), case["fp64"]), device="cuda")


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case)
    if kind == "layer":
        s["psi"], s["bonds"], s["gates"], s["sites"], s["u"] = _layer_inputs(case, seed)
        s["engine"] = mg.Engine(fp64=case["fp64"])
        s["engine"].adopt(s["psi"].data_ptr(), case["n"])
    elif kind in ("entropy", "rho3"):
        s["psi"] = _trajectory_state(case["n"], seed, case["fp64"])
    elif kind == "batch":
        s["seeds"], s["p"] = np.array(_seeds(seed, case["count"]), np.uint64), _p_of(case)
        s["batch"] = _make_batch(case)
    elif kind == "free":
        s["initial"] = np.array(_seeds(seed, case["count"]), np.uint64)
        s["workspace"] = np.array(_seeds(seed + 1, case["count"], 32), np.uint32)
        s["batch"] = mg.Batch(case["n"], case["layers"] // 2, case["count"], closed=True, fp64=case["fp64"],
                              observables=mg.OBS_SVN_HALF)
        s["batch"].set_observation_steps(list(range(case["points"])))
    elif kind == "ff":
        s["seeds"] = np.array(_seeds(seed, case["count"]), np.uint64)
    else:
        s["rho"] = _three_qubit_states(case, seed)
    return s


def run(state):
    case = state["case"]
    kind, fp64 = case["kind"], case.get("fp64", True)
    if kind == "layer":
        e = state["engine"]
        e.apply_bonds(state["bonds"], state["gates"])
        outcomes, surprisal = e.measure_layer(state["sites"], state["u"])
        return dict(state=state["psi"], outcomes=outcomes, surprisal=_real(surprisal, fp64))
    if kind == "entropy":
        f = mg.entropy_svd if case["order"] == 1 else mg.renyi2
        return _real(f(state["psi"].data_ptr(), case["n"], _kept(case), fp64=fp64), fp64)
    if kind == "rho3":
        return _real(mg.rho3_subsystems(state["psi"].data_ptr(), case["n"], _ring(case["n"]), fp64=fp64), fp64)
    if kind == "batch":
        b = state["batch"]
        r = b.run(state["seeds"], state["p"])
        out = dict(outcomes=r["outcomes"].view(np.int64), surprisal=_real(r["surprisal"], fp64),
                   state=_batch_states(b, case))
        for i, want in enumerate(("svn", "s2", "tmi_vn", "tmi_s2")):
            if case[want]:
                out[want] = _real(r["obs"][:, :, i], fp64)
        if case["region"]:
            out["region"] = _real(b.fetch_regions()[:, :, 0], fp64)
        if case["rho3"]:
            out["rho3"] = _real(r["rho3"], fp64)
        return out
    if kind == "free":
        b = state["batch"]
        b.set_initial_states(state["initial"], 0)
        b.prepare_workspace(state["workspace"], case["p"])
        b.execute()
        r = b.fetch()
        return dict(outcomes=r["outcomes"].view(np.int64), surprisal=_real(r["surprisal"], fp64),
                    svn=_real(r["obs"][:, :, 0], fp64), state=_batch_states(b, case))
    if kind == "ff":
        r = mg.ff_run(state["seeds"], case["p"], case["n"], case["depth"], closed=case["closed"],
                      repurify_every=case["every"], blocks=_blocks(case["n"]), want_gamma=True, fp64=fp64)
        return dict(outcomes=r["outcomes"], probs=_real(r["probs"], fp64), gamma=_real(r["gamma"], fp64),
                    blocks=_real(r["s_blocks"], fp64), tmi=_real(r["tmi"], fp64))
    r = mg.gmn_solve(state["rho"], gap_tol=1e-6, max_iter=case["max_iter"], check_every=10, fp64=fp64)
    return dict(gmn=_real(r["gmn"], fp64), gap=_real(r["gap"], fp64), iterations=r["iters"])


def _regions(case):
    """(name, kept, order) of a chain batch's observables; TMI parts carry a sign."""
    n, q = case["n"], case["n"] // 4
    half = list(range(n // 2))
    parts = [list(range(i * q, (i + 1) * q)) for i in range(4)]
    signed = [(1, x) for x in parts] + [(-1, parts[0] + parts[1]), (-1, parts[0] + parts[2]), (-1, parts[1] + parts[2])]
    out = []
    if case.get("svn", True):
        out.append(("svn", 1, [(1, half)]))
    if case.get("s2"):
        out.append(("s2", 2, [(1, half)]))
    if case.get("tmi_vn"):
        out.append(("tmi_vn", 1, signed))
    if case.get("tmi_s2"):
        out.append(("tmi_s2", 2, signed))
    if case.get("region"):
        out.append(("region", 1, [(1, list(range(case["region"])))]))
    return out


def _points(case):
    layers = 2 * case["periods"] + (case["circuit"] in (2, 4))
    return [layers] if not case["every"] else list(range(case["every"], layers + 1, case["every"]))


def work(case):
    """Bytes: a layer's state is read and written once, inputs and outputs
    once. Flops: 8 per complex multiply-add of gates (16 real multiply-adds
    per amplitude and bond), Gram matrices on the smaller side, 16/3 d^3 per
    Hermitian spectrum."""
    kind, n = case["kind"], case.get("n", 3)
    amp = 16.0 if case.get("fp64") else 8.0
    dim = float(1 << n) if kind != "ff" else 0.0

    def observed(order, k):
        d = 2.0 ** min(k, n - k)
        return 2 * _gram_work(n, k) + (16.0 / 3.0 * d ** 3 if order == 1 else 0.0)

    if kind == "layer":
        return dict(bytes=2 * dim * amp, flops=32.0 * dim * len(_bonds(n, case["odd"], case["closed"])))
    if kind == "entropy":
        return dict(bytes=dim * amp, flops=observed(case["order"], case["k"]))
    if kind == "rho3":
        return dict(bytes=dim * amp, flops=n * 8.0 * 8 * dim)
    if kind in ("batch", "free"):
        layers = case["layers"] if kind == "free" else 2 * case["periods"]
        points = case["points"] if kind == "free" else len(_points(case))
        flops = case["count"] * (layers * 32.0 * dim * (n // 2)
                                 + points * sum(observed(o, len(x)) for _, o, v in _regions(case) for _, x in v))
        return dict(bytes=case["count"] * layers * 2 * dim * amp, flops=flops)
    if kind == "ff":
        size = 4.0 * n * n
        per_layer = 16.0 * size / 2 + case["p"] * n * 4.0 * size / 2
        real = 8.0 if case["fp64"] else 4.0
        blocks = sum(8.0 / 3.0 * (2.0 * b) ** 3 for b in _blocks(n) + [n // 4] * 4 + [n // 2] * 3)
        purify = 2 * 2 * (2.0 * n) ** 3 * (1 + (case["depth"] // case["every"] if case["every"] else 0))
        return dict(bytes=case["count"] * size * (8.0 + real), flops=case["count"] * (case["depth"] * per_layer + blocks
                                                                                     + purify))
    # About 40 iterations, six 8 x 8 complex eigenproblems each.
    return dict(bytes=case["count"] * (1024.0 + 20.0), flops=case["count"] * 40 * 6 * 20.0 * 8 ** 3)


# --------------------------------------------------------------- in 64 bits
def _exact_batch(case, seed):
    n, count = case["n"], case["count"]
    layers = 2 * case["periods"]
    if case["circuit"] != 1 or count * layers * (1 << n) > EVOLVE_LIMIT:
        return None
    points = _points(case)
    out = dict(outcomes=None, surprisal=np.zeros((count, layers)))
    out.update({name: None for name, _, _ in _regions(case)})
    wanted = []
    for name, order, parts in _regions(case):
        total = count * len(points)
        gram = total * sum(_gram_work(n, len(x)) for _, x in parts)
        eig = total * sum(8.0 ** min(len(x), n - len(x)) for _, x in parts) if order == 1 else 0
        if gram < GRAM_LIMIT and eig < EIG_LIMIT:
            wanted.append((name, order, parts))
            out[name] = np.zeros((count, len(points)))
    out["state"] = torch.zeros((count, 1 << n), dtype=torch.complex128, device=_device())
    for i, (sd, p) in enumerate(zip(_seeds(seed, count), _p_of(case))):
        psi = torch.zeros(1 << n, dtype=torch.complex128, device=_device())
        psi[0] = 1
        seen = []
        for t, layer in enumerate(_haar_record(sd, n, layers, p, case["closed"], case["lattice_x"])):
            _, out["surprisal"][i, t], psi = _layer(psi, n, layer)
            if t + 1 in points and wanted:
                seen.append(psi)
        for name, order, parts in wanted:
            step = max(1, (1 << 26) >> n)
            for j in range(0, len(seen), step):
                v = sum(sign * _entropy(torch.stack(seen[j:j + step]), n, x, order) for sign, x in parts)
                out[name][i, j:j + step] = v.cpu().numpy()
        out["state"][i] = psi
    if case["rho3"]:
        out["rho3"] = np.stack([np.concatenate([_rho3(x, n, t) for t in _triples(case)]).reshape(-1, 128)
                                for x in out["state"]])
    return out


def _rho3(psi, n, triple):
    m = _rows(psi, n, triple)
    return torch.view_as_real(m @ m.transpose(-1, -2).conj()).reshape(-1).cpu().numpy()


def _exact_free(case, seed):
    n, count, layers = case["n"], case["count"], case["layers"]
    points = case["points"]
    out = dict(outcomes=None, surprisal=np.zeros((count, layers)), svn=None,
               state=torch.zeros((count, 1 << n), dtype=torch.complex128, device=_device()))
    if count * points * 8.0 ** (n // 2) < EIG_LIMIT:
        out["svn"] = np.zeros((count, points))
    for i, (a, w) in enumerate(zip(_seeds(seed, count), _seeds(seed + 1, count, 32))):
        psi = torch.as_tensor(_product_state(a, n, case["fp64"]), device=_device()).to(torch.complex128)
        seen = [psi]
        for t, layer in enumerate(_haar_record(w, n, layers, case["p"], True, workspace=True)):
            _, out["surprisal"][i, t], psi = _layer(psi, n, layer)
            if t + 1 < points:
                seen.append(psi)
        if out["svn"] is not None:
            out["svn"][i] = _entropy(torch.stack(seen), n, list(range(n // 2)), 1).cpu().numpy()
        out["state"][i] = psi
    return out


def _ff_record(seed, n, depth, p, closed):
    gates, meas = _Stream(seed), _Stream(_splitmix64(seed ^ 0xA0761D0D))
    out = []
    for t in range(depth):
        modes = [a for a, _ in _bonds(n, t % 2 == 1, closed)]
        q = _gram_schmidt(np.swapaxes(gates.normals(16 * len(modes)).reshape(-1, 4, 4), 1, 2))
        q[np.linalg.det(q) < 0, :, 0] *= -1
        sites = np.nonzero(gates.take(n) < p)[0]
        out.append((modes, q, sites, meas.take(len(sites))))
    return out


def _repurified(g):
    return 1.5 * g + 0.5 * g @ g @ g


def _ff_entropy(g, modes):
    """Block entropy from the positive half of i Gamma's spectrum."""
    idx = torch.as_tensor([2 * m + j for m in modes for j in (0, 1)], device=g.device)
    nu = torch.linalg.eigvalsh(1j * g[:, idx][:, :, idx])[:, len(modes):].clamp(0.0, 1.0)
    s = 0.0
    for x in ((1 + nu) / 2, (1 - nu) / 2):
        s = s + torch.where(x > 1e-15, -x * torch.log2(x.clamp_min(1e-300)), torch.zeros_like(x)).sum(1)
    return s


def _exact_ff(case, seed):
    n, depth, count = case["n"], case["depth"], case["count"]
    dev = _device()
    records = [_ff_record(sd, n, depth, case["p"], case["closed"]) for sd in _seeds(seed, count)]
    g = torch.zeros((count, 2 * n, 2 * n), dtype=torch.float64, device=dev)
    even = torch.arange(0, 2 * n, 2, device=dev)
    g[:, even, even + 1], g[:, even + 1, even] = 1, -1
    probs = np.zeros((count, depth, n))
    every = torch.arange(count, device=dev)
    for t in range(depth):
        o = torch.eye(2 * n, dtype=torch.float64, device=dev).repeat(count, 1, 1)
        rot = torch.as_tensor(np.stack([r[t][1] for r in records]), device=dev)
        for j, m in enumerate(records[0][t][0]):
            idx = torch.as_tensor([2 * m, 2 * m + 1, 2 * ((m + 1) % n), 2 * ((m + 1) % n) + 1], device=dev)
            o[:, idx[:, None], idx[None, :]] = rot[:, j]
        g = o @ g @ o.transpose(1, 2)
        for i in range(max(len(r[t][2]) for r in records)):
            who = torch.as_tensor([c for c in range(count) if i < len(records[c][t][2])], device=dev)
            a = torch.as_tensor([2 * int(records[c][t][2][i]) for c in who.tolist()], device=dev)
            u = torch.as_tensor([records[c][t][3][i] for c in who.tolist()], device=dev, dtype=torch.float64)
            at = every[: len(who)]
            x = g[who]
            v = x[at, a, a + 1]
            up = ((1 + v) / 2).clamp(0, 1)
            s = torch.where(u < up, 1.0, -1.0).to(torch.float64)
            probs[who.cpu().numpy(), t, i] = torch.where(s > 0, up, 1 - up).cpu().numpy()
            ua, vb = x[at, :, a].clone(), x[at, :, a + 1].clone()
            x = x + (vb[:, :, None] * ua[:, None, :] - ua[:, :, None] * vb[:, None, :]) / (v + s)[:, None, None]
            for b in (a, a + 1):
                x[at, b, :], x[at, :, b] = 0, 0
            x[at, a, a + 1], x[at, a + 1, a] = s, -s
            g[who] = x
        if case["every"] and (t + 1) % case["every"] == 0:
            g = _repurified(g)
    q = n // 4
    part = [list(range(i * q, (i + 1) * q)) for i in range(4)]
    tmi = (sum(_ff_entropy(g, x) for x in part) - _ff_entropy(g, part[0] + part[1])
           - _ff_entropy(g, part[0] + part[2]) - _ff_entropy(g, part[1] + part[2]))
    return dict(outcomes=None, probs=probs, gamma=g, tmi=tmi.cpu().numpy(),
                blocks=np.stack([_ff_entropy(g, list(range(b))).cpu().numpy() for b in _blocks(n)], 1))


def exact(case, seed):
    kind, n = case["kind"], case.get("n", 0)
    if kind == "layer":
        psi, bonds, gates, sites, u = _layer_inputs(case, seed)
        _, surprisal, psi = _layer(psi.to(torch.complex128), n, (bonds, gates, sites, u))
        return dict(state=psi, outcomes=None, surprisal=np.float64(surprisal))
    if kind == "entropy":
        psi = _trajectory_state(n, seed, case["fp64"]).to(torch.complex128)
        return _entropy(psi, n, _kept(case), case["order"]).cpu().numpy()
    if kind == "rho3":
        psi = _trajectory_state(n, seed, case["fp64"]).to(torch.complex128)
        return np.concatenate([_rho3(psi, n, t) for t in _ring(n)])
    if kind == "batch":
        return _exact_batch(case, seed)
    if kind == "free":
        return _exact_free(case, seed)
    if kind == "ff":
        return _exact_ff(case, seed) if case["count"] * case["depth"] * case["n"] ** 3 < 5e10 else None
    return None  # an iterate of a first-order method: no closed form
