"""Performance cases of the adaptive-basis time step: what programs on this framework spend
their time in, from the smallest chains to the 2^22-state ring.

A case is one call of the engine's public entry points on a state that has already spread:

  step    `Trajectory.step`, one evolving time step (truncate, enlarge, assemble H, carry the
          amplitudes over, propagate, observables), by the Taylor series, by Lanczos
          (`lanczos` > 0) or by scaling and squaring (`scaled`)
  batch   `TrajectoryBatch.step`, several trajectories advanced together
  expand  `Engine.expand`, the enlargement that grows a basis before a run

A step only reads the old state, so the same step can be taken again from the same slot.

States are made here with plain torch, from the seed alone: a phonon cloud around an exciton
wave packet ranks the states, the basis is grown and cut by that rank as a run grows and cuts
it, and the amplitudes get random phases and a spread of magnitudes.  The state at which a
step starts is, as in a run, the truncated basis with everything two applications of H reach
(enlarge_steps + 1 in general).
"""

import math

import numpy as np
import torch

DEV = "cuda"
SIGN = -(1 << 63)
ROUNDS_AT_CUT = 3  # truncate-and-grow rounds after the basis has reached maxstates

DEFAULTS = dict(kind="step", nchain=32, dim=16, precision="c128", g=1.5, hbar_omega=1.0, eps_sys=0.0, J2=0.0,
                geo_dim=1, periodic=True, sigma=0.0, maxstates=1 << 16, enlarge_steps=1, dt=0.05, graph=False,
                lanczos=0, weighting="none", tau=0.0, scaled=False, trajectories=1)


def listed():
    return [
        # the benchmark's ring in single precision: a long production run, every step replayed as a CUDA graph
        dict(name="ring32_c64_4m", precision="c64", maxstates=1 << 22, graph=True),
        # the same physics in the reference's own precision, as a driver script of the reference runs it
        dict(name="ring32_c128_1m", maxstates=1 << 20),
        # mid-sized open chain: the reference's only boundary; parameter scans at 2^16 states
        dict(name="chain16_c128_64k", nchain=16, g=1.0, periodic=False, sigma=0.1, maxstates=1 << 16),
        # smallest: short chains of convergence checks, where launches and waits are what a step costs
        dict(name="chain8_c128_4k", nchain=8, g=1.0, periodic=False, maxstates=4001),
        # long disordered chain (four key words), small time step
        dict(name="chain64_c64_512k", nchain=64, g=2.0, precision="c64", sigma=0.5, maxstates=(1 << 19) + 77, dt=0.025,
             graph=True),
        # the reference's example driver: 25 sites, 128 levels (7-bit fields, three key words), strong coupling
        dict(name="example25_c128_300k", nchain=25, dim=128, g=4.0, eps_sys=-1.0, periodic=False, maxstates=300001),
        # Krylov propagation (ExpmParams.lanczos_order) of a ring
        dict(name="lanczos24_c128_200k", nchain=24, maxstates=200003, lanczos=12),
        # square lattice with next-nearest hopping, 4 levels per site (one key word of 2-bit fields)
        dict(name="lattice16_c128_100k", nchain=16, dim=4, g=1.0, geo_dim=2, J2=0.5, periodic=False, maxstates=100003),
        # look-ahead weighting in the truncation
        dict(name="coherence32_c128_256k", maxstates=1 << 18, weighting="coherence", tau=0.2),
        # scaling and squaring (ExpmParams.use_scaling)
        dict(name="scaled16_c128_50k", nchain=16, g=1.0, periodic=False, maxstates=50001, scaled=True),
        # a parameter scan advanced together: rings of 16, 24 and 32 sites, each with its own g, omega and size
        dict(name="batch8_c64", kind="batch", precision="c64", maxstates=1 << 17, trajectories=8, graph=True),
        # growing the starting basis of a large run
        dict(name="grow32_c128_1m", kind="expand", maxstates=(1 << 20) + 5),
    ]


def draw(rng):
    """One more case of the same ranges: any boundary, field width, precision, propagator and size."""
    kind = rng.choices(["step", "batch", "expand"], [8, 1, 1])[0]
    c = dict(kind=kind, precision=rng.choice(["c64", "c128"]), g=round(rng.uniform(0.5, 2.0), 3),
             hbar_omega=round(rng.uniform(0.5, 1.5), 3), graph=rng.random() < 0.5)
    c["nchain"] = rng.choice([rng.randint(8, 16), rng.randint(17, 32), rng.randint(33, 64)])
    c["dim"] = rng.choice([16, 16, rng.choice([8, 12, 32, 128])])
    c["periodic"] = rng.random() < 0.5
    c["sigma"] = rng.choice([0.0, 0.5])
    words = -(-c["nchain"] // (64 // max(1, (c["dim"] - 1).bit_length())))
    most = 21.0 if words <= 2 else (20.0 if words <= 4 else 19.0)
    c["maxstates"] = int(2.0 ** rng.uniform(11.0, most))
    if kind == "batch":
        c.update(trajectories=rng.randint(2, 12), maxstates=int(2.0 ** rng.uniform(12.0, 17.0)), sigma=0.0,
                 periodic=True, dim=16, nchain=32)
    if kind == "step":
        c["enlarge_steps"] = rng.choices([1, 0, 2], [6, 1, 1])[0]
        c["maxstates"] >>= 1 if c["enlarge_steps"] == 2 else 0
        c["dt"] = rng.choice([0.05, 0.025, 0.1])
        what = rng.choices(["taylor", "lanczos", "scaled", "weighted", "lattice"], [8, 1, 1, 1, 1])[0]
        if what == "lanczos":
            c.update(lanczos=rng.choice([8, 12, 20]), maxstates=min(c["maxstates"], 1 << 19))
        elif what == "scaled":
            c.update(scaled=True, precision="c128")
        elif what == "weighted":
            c.update(weighting=rng.choice(["coherence", "norm"]), tau=0.2, precision="c128")
        elif what == "lattice":
            c.update(geo_dim=2, nchain=rng.choice([9, 16, 25]), dim=rng.choice([4, 8, 16]), J2=rng.choice([0.0, 0.5]),
                     periodic=False, maxstates=min(c["maxstates"], 1 << 19))
    return c


# ---- plain torch: packed states, images, sorted sets ------------------------------------------
def _full(case):
    c = dict(DEFAULTS)
    c.update(case)
    return c


def _members(case, seed):
    """The parameters of every trajectory of a case (one, or a batch's), with its site energies."""
    c = _full(case)
    rng = np.random.default_rng([int(seed), 11])
    out = []
    for k in range(c["trajectories"]):
        m = dict(c)
        if c["kind"] == "batch":
            m.update(nchain=int((16, 24, 32)[k % 3]), g=float(rng.uniform(0.5, 2.0)),
                     hbar_omega=float(rng.uniform(0.5, 1.5)),
                     maxstates=int(c["maxstates"] * 2.0 ** (-3.0 * ((k * 5) % 8) / 8.0)) + k)
        m["site_eps"] = None
        if m["sigma"] > 0:
            m["site_eps"] = [float(x) for x in rng.normal(0.0, m["sigma"], m["nchain"])]
        m["seed"] = int(seed) * 64 + k
        out.append(m)
    return out


class Space:
    """The packing of a model's states (most significant field first, fields never straddle a
    64-bit word) and its images under H."""

    def __init__(self, m):
        self.m = m
        self.L, self.dim = m["nchain"], m["dim"]
        self.bits = max(1, (self.dim - 1).bit_length())
        self.fpw = 64 // self.bits
        self.nw = -(-self.L // self.fpw)
        self.mask = (1 << self.bits) - 1
        s = torch.arange(self.L, device=DEV)
        self.word = s // self.fpw
        self.shift = 64 - self.bits * (s % self.fpw + 1)
        l = round(self.L ** (1.0 / m["geo_dim"]))
        self.hops = []  # distance, lattice period, matrix element
        for order, amp in ((1, 1.0), (2, m["J2"])):
            if order == 1 or amp != 0.0:
                self.hops += [(order * l ** d, l ** (d + 1), amp) for d in range(m["geo_dim"])]

    def field(self, words, s):
        return (words[s // self.fpw] >> (64 - self.bits * (s % self.fpw + 1))) & self.mask

    def own(self, pos, words):
        """Occupation of the exciton's own site."""
        w = words[0].clone()
        for q in range(1, self.nw):
            w = torch.where(self.word[pos] == q, words[q], w)
        return (w >> self.shift[pos]) & self.mask

    def images(self, pos, words):
        """Per coupling the images: (exists, position, words)."""
        out = []
        for d, md, _ in self.hops:
            for up in (0, 1):
                if self.m["periodic"]:
                    ok, q = torch.ones_like(pos, dtype=torch.bool), (pos + (d if up else self.L - d)) % self.L
                else:
                    ok, q = (pos % md < md - d, pos + d) if up else (pos % md >= d, pos - d)
                out.append((ok, q, words))
        n = self.own(pos, words)
        one = torch.ones_like(pos) << self.shift[pos]
        at = [(self.word[pos] == q).to(torch.int64) * one for q in range(self.nw)]
        out.append((n > 0, pos, [w - a for w, a in zip(words, at)]))
        out.append((n + 1 < self.dim, pos, [w + a for w, a in zip(words, at)]))
        return out

    @staticmethod
    def order(pos, words):
        idx = None
        for k in [w ^ SIGN for w in reversed(words)] + [pos]:
            k = k if idx is None else k[idx]
            o = torch.sort(k, stable=True)[1]
            idx = o if idx is None else idx[o]
        return idx

    def unique(self, pos, words):
        """Sorted distinct states and the index of every input among them."""
        idx = self.order(pos, words)
        pos, words = pos[idx], [w[idx] for w in words]
        new = torch.ones_like(pos, dtype=torch.bool)
        new[1:] = pos[1:] != pos[:-1]
        for w in words:
            new[1:] |= w[1:] != w[:-1]
        rank = torch.empty_like(idx)
        rank[idx] = torch.cumsum(new, 0) - 1
        return pos[new], [w[new] for w in words], rank

    def grow(self, pos, words, table=False):
        """The states with all their images; with `table` also each state's neighbours: for
        every coupling in the order of images(), the index of its image or -1 (a coupling is
        in H when one of its two states is among the given ones)."""
        ims = self.images(pos, words)
        p = torch.cat([pos] + [q[ok] for ok, q, _ in ims])
        w = [torch.cat([words[k]] + [iw[k][ok] for ok, _, iw in ims]) for k in range(self.nw)]
        np_, nw_, rank = self.unique(p, w)
        if not table:
            return np_, nw_, None
        src, off = rank[:pos.numel()], pos.numel()
        nbr = torch.full((len(ims), np_.numel()), -1, dtype=torch.int64, device=DEV)
        for k, (ok, _, _) in enumerate(ims):
            n = int(ok.sum())
            to = rank[off:off + n]
            off += n
            nbr[k, src[ok]] = to
            nbr[k ^ 1, to] = src[ok]  # images() lists every coupling beside its reverse
        return np_, nw_, nbr

    def phonons(self, words):
        return sum(self.field(words, s) for s in range(self.L))

    def log_weight(self, pos, words, x0):
        """Rank of a state: phonon clouds (displaced oscillators, narrowing with the distance from
        the exciton) under an exponential exciton envelope."""
        g = max(self.m["g"], 0.3)
        dist = torch.arange(self.L, device=DEV)
        if self.m["periodic"]:
            dist = torch.minimum(dist, self.L - dist)
        lg = torch.lgamma(torch.arange(self.dim, device=DEV, dtype=torch.float64) + 1.0) * 0.5
        cloud = torch.log(g * torch.exp(-0.6 * dist.double()) + 0.04)
        out = -0.25 * dist[(pos - x0).abs()].double()
        for s in range(self.L):
            n = self.field(words, s)
            out += n * cloud[(pos - s).abs()] - lg[n]
        h = pos * 0x9E3779B97F4A7C1 + self.m["seed"]  # a state's own deviation: no two states tie
        for w in words:
            h = (h ^ w) * 0x2545F4914F6CDD1D
            h = h ^ ((h >> 29) & 0x7FFFFFFFF)
        return out + 0.2 * ((h >> 11) & 0xFFFFFFFFFF).double() / float(1 << 40)

    def diagonal(self, pos, words):
        d = self.m["eps_sys"] + self.m["hbar_omega"] * self.phonons(words).double()
        if self.m["site_eps"] is not None:
            d = d + torch.tensor(self.m["site_eps"], device=DEV, dtype=torch.float64)[pos]
        return d


def _start(m):
    """A model's spread state: (space, positions, words, amplitudes complex128)."""
    sp = Space(m)
    gen = torch.Generator(device=DEV)
    gen.manual_seed(m["seed"] * 7919 + 17)
    x0 = int(np.random.default_rng([m["seed"], 5]).integers(0, sp.L))
    pos = torch.tensor([x0], device=DEV)
    words = [torch.zeros(1, dtype=torch.int64, device=DEV) for _ in range(sp.nw)]
    M, cuts = m["maxstates"], 0
    while True:
        n0 = pos.numel()
        p, w, _ = sp.grow(pos, words)
        if p.numel() > M:
            top = torch.topk(sp.log_weight(p, w, x0), M, sorted=False)[1].sort()[0]
            p, w = p[top], [x[top] for x in w]
            cuts += 1
        pos, words = p, w
        if cuts >= ROUNDS_AT_CUT or (cuts == 0 and pos.numel() == n0):
            break
    if m["kind"] == "expand":
        return sp, pos, words, None
    for _ in range(m["enlarge_steps"] + 1):
        pos, words, _ = sp.grow(pos, words)
    n = pos.numel()
    mag = torch.exp(sp.log_weight(pos, words, x0) + 0.3 * torch.randn(n, generator=gen, device=DEV, dtype=torch.float64))
    if n > M:  # a clear cut at maxstates: no two nearly equal magnitudes on either side of it
        cut = torch.topk(mag, M)[0][-1]
        mag = torch.where(mag < cut, mag * 0.999, mag)
    ph = torch.rand(n, generator=gen, device=DEV, dtype=torch.float64) * (2.0 * math.pi)
    psi = torch.polar(mag / torch.linalg.vector_norm(mag), ph)
    return sp, pos, words, psi


# ---- the calls ---------------------------------------------------------------------------------
def _engine(m, cap):
    from paces_b200.engine import Engine, ModelParams
    return Engine(ModelParams(nchain=m["nchain"], max_ho_dims=[m["dim"]] * m["nchain"], J=1.0, g=m["g"],
                              eps_sys=m["eps_sys"], hbar_omega=m["hbar_omega"], periodic=m["periodic"],
                              site_eps=m["site_eps"], precision=m["precision"], geo_dim=m["geo_dim"],
                              J2=m["J2"] if m["J2"] else None), cap=cap)


def _basis(eng, sp, pos, words):
    b = eng.new_basis(pos.numel())
    b.keys.copy_(torch.stack(words, dim=1))
    b.blk[1:] = torch.cumsum(torch.bincount(pos, minlength=sp.L), 0).to(torch.int32)
    return b


def _room(m):
    """States to have room for: the next step's basis as well, as in a run that has grown to its size."""
    if m["kind"] == "expand":
        return 7 * m["maxstates"] + 4096
    per = (4.5, 7, 12)[m["enlarge_steps"]] * (2 if m["geo_dim"] > 1 else 1)
    return int(per * m["maxstates"]) + 4096


def prepare(case, seed):
    from paces_b200 import _native as nat
    from paces_b200.engine import Trajectory, TrajectoryBatch
    c = _full(case)
    trajs = []
    for m in _members(case, seed):
        sp, pos, words, psi = _start(m)
        if c["kind"] == "expand":
            eng = _engine(m, _room(m))
            out = eng.new_basis()
            out.keys.zero_()
            return dict(case=c, eng=eng, basis=_basis(eng, sp, pos, words), out=out)
        eng = _engine(m, 4096)
        kind = {"none": nat.WEIGHT_NONE, "coherence": nat.WEIGHT_COHERENCE, "norm": nat.WEIGHT_NORM}[m["weighting"]]
        tr = Trajectory(eng, m["maxstates"], m["enlarge_steps"], cap=_room(m), graph=m["graph"], weighting=kind,
                        tau=m["tau"], lanczos_order=m["lanczos"])
        for b, h in zip(tr.bases, tr.hs):  # the rows past a basis' last state stay zero
            for t in (b.keys, h.nbr, h.meta) + (() if h.xnbr is None else (h.xnbr,)):
                t.zero_()
        tr.set_state(_basis(eng, sp, pos, words), psi)
        if m["scaled"]:  # that step uses the old slot's amplitudes as scratch: the program sets the state again
            return dict(case=c, trajs=[tr], basis=_basis(eng, sp, pos, words), psi=psi)
        if kind:  # the weights come from the table of the state's own basis: a first, non-evolving step
            tr.step(evolve=False)
        trajs.append(tr)
    state = dict(case=c, trajs=trajs, slots=[t.cur for t in trajs])
    if c["kind"] == "batch":
        state["batch"] = TrajectoryBatch(trajs, graph=c["graph"])
    return state


def _result(tr, rec):
    """The new state in its buffers (states 0 .. blk[-1]) and its observables."""
    L = tr.eng.L
    out = {"keys": tr.basis.keys, "blk": tr.basis.blk, "nbr": tr.h.nbr, "meta": tr.h.meta,
           "psi": tr.psis[tr.cur], "n_exc": np.array(rec.n_exc[:L]), "n_pho": np.array(rec.n_pho[:L]),
           "norm_energy": np.array([rec.norm, rec.energy_re])}
    if tr.h.xnbr is not None:
        out["xnbr"] = tr.h.xnbr
    return out


def run(state):
    c = state["case"]
    if c["kind"] == "expand":
        b = state["eng"].expand(state["basis"], state["out"])
        return {"keys": b.keys, "blk": b.blk}
    if c["scaled"]:
        tr = state["trajs"][0]
        tr.set_state(state["basis"], state["psi"])
        return _result(tr, tr.step_scaled(c["dt"]))
    for t, slot in zip(state["trajs"], state["slots"]):
        t.cur = slot  # the old state is as it was: the step starts from it again
    if c["kind"] == "batch":
        recs = state["batch"].step(True, c["dt"])
        out = [_result(t, r) for t, r in zip(state["trajs"], recs)]
        return [{k: o[k] for k in ("keys", "psi", "nbr", "n_pho", "norm_energy")} for o in out]
    tr = state["trajs"][0]
    return _result(tr, tr.step(True, c["dt"]))


def work(case):
    """Bytes: the old state's keys and amplitudes in, the new state's keys, table and amplitudes
    out.  Operations: the rows of H once per Taylor term or Krylov vector.  A new basis holds
    about 4 maxstates states at enlarge_steps 1 (2 at 0, 7 at 2; 9 on a square lattice)."""
    c = _full(case)
    nbytes = flops = 0.0
    for m in _members(case, 0):
        kb = 8 * -(-m["nchain"] // (64 // max(1, (m["dim"] - 1).bit_length())))
        if c["kind"] == "expand":
            nbytes += 3.1 * m["maxstates"] * kb
            continue
        S = m["maxstates"] * (9.0 if m["geo_dim"] > 1 else {0: 2.0, 1: 4.0, 2: 7.0}[m["enlarge_steps"]])
        cs = 8 if m["precision"] == "c64" else 16
        nbytes += S * 2 * (kb + cs) + S * 20
        terms = m["lanczos"] or (8 if m["precision"] == "c64" else 15)
        flops += S * terms * 34
    return {"bytes": nbytes, "flops": flops}


# ---- the same in 64 bits, with plain torch -----------------------------------------------------
class _Ham:
    def __init__(self, sp, pos, words, nbr):
        self.sp, self.pos, self.words, self.nbr = sp, pos, words, nbr
        self.diag = sp.diagonal(pos, words)
        n = sp.own(pos, words).double()
        self.amps = [a for _, _, a in sp.hops for _ in (0, 1)]
        self.amps += [sp.m["g"] * torch.sqrt(n), sp.m["g"] * torch.sqrt(n + 1.0)]

    def apply(self, x):
        y = self.diag * x
        for k, amp in enumerate(self.amps):
            j = self.nbr[k]
            y += torch.where(j >= 0, x[j.clamp(min=0)], 0.0) * amp
        return y

    def ones(self):
        y = self.diag.clone()
        for k, amp in enumerate(self.amps):
            y += (self.nbr[k] >= 0).double() * amp
        return y


def _adapt(sp, pos, words, psi, weight, M, enlarge_steps):
    """Truncate by weight, enlarge, take everything H reaches, carry the amplitudes over."""
    p, w = pos, words
    if pos.numel() > M:
        top = torch.topk(weight, M, sorted=False)[1].sort()[0]
        p, w = pos[top], [x[top] for x in words]
    for _ in range(enlarge_steps):
        p, w, _ = sp.grow(p, w)
    p, w, nbr = sp.grow(p, w, table=True)
    _, _, rank = sp.unique(torch.cat([p, pos]), [torch.cat([a, b]) for a, b in zip(w, words)])
    n = p.numel()
    amp = torch.zeros(int(rank.max()) + 1, dtype=torch.complex128, device=DEV)
    amp[rank[n:]] = psi
    return p, w, nbr, amp[rank[:n]]


def _exact_one(m):
    sp, pos, words, psi = _start(m)
    psi = psi.to(torch.complex64 if m["precision"] == "c64" else torch.complex128).to(torch.complex128)
    M, es = m["maxstates"], m["enlarge_steps"]
    weight = psi.abs()
    if m["weighting"] != "none":
        pos, words, nbr, psi = _adapt(sp, pos, words, psi, weight, M, es)
        h = _Ham(sp, pos, words, nbr)
        if m["weighting"] == "coherence":
            p2 = psi.real ** 2 + psi.imag ** 2
            weight = p2 + m["tau"] ** 2 * p2 * h.ones() ** 2
        else:
            weight = (psi - 1j * m["tau"] * h.apply(psi)).abs()
        del h, nbr
    pos, words, nbr, psi = _adapt(sp, pos, words, psi, weight, M, es)
    h = _Ham(sp, pos, words, nbr)
    factor = (1j if m["scaled"] else -1j) * m["dt"]  # scaling and squaring propagates with +1j H
    term, out = psi, psi.clone()
    for k in range(1, 120):
        term = h.apply(term) * (factor / k)
        out += term
        if float(term.abs().max()) < 1e-20:
            break
    w = out.real ** 2 + out.imag ** 2
    energy = float((out.conj() * h.apply(out)).real.sum())
    n_exc = torch.zeros(sp.L, dtype=torch.float64, device=DEV).index_add_(0, pos, w)
    n_pho = torch.stack([(w * sp.field(words, s)).sum() for s in range(sp.L)])
    psi = torch.zeros(_room(m), dtype=torch.complex128, device=DEV)
    psi[:out.numel()] = out
    return {"keys": None, "blk": None, "nbr": None, "meta": None, "psi": psi, "n_exc": n_exc.cpu().numpy(),
            "n_pho": n_pho.cpu().numpy(), "norm_energy": np.array([math.sqrt(float(w.sum())), energy])}


def exact(case, seed):
    c = _full(case)
    if c["kind"] == "expand":
        return None
    out = [_exact_one(m) for m in _members(case, seed)]
    if c["kind"] == "batch":
        return [{k: o[k] for k in ("keys", "psi", "nbr", "n_pho", "norm_energy")} for o in out]
    if c["geo_dim"] > 1:
        out[0]["xnbr"] = None
    return out[0]
