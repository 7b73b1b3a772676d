"""What a user of this engine has it do, as measurable cases.

Every case is one call (or the few calls a program makes together) through the
package's public entry points: ``Hamiltonian.apply_within`` with and without
its backward, ``diagonal_term``, ``find_relative``, ``single_relative_seeded``,
``variational_energy`` with its gradient, ``lanczos_energy``, ``pt2_energy``
and the network sampler's ``generate_unique``.  Sizes are those of the
benchmark's workloads and of the tests, or lie between them.

A Hamiltonian is kept per molecule or lattice (a program compiles it once and
then calls it on ever new configurations); configurations, amplitudes and
everything else a call takes come from the case's seed.
"""

from __future__ import annotations

import functools
import importlib
import math

import numpy as np
import torch

qmb = importlib.import_module("qmb-public_gb300")


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------

_LISTED = [
    # the smallest call: H psi and the diagonal over every determinant of 12 spin orbitals (an
    # exact diagonalisation's inner call); launches and the host path are all there is
    dict(name="exact_12", kind="apply", orbits=6, alpha=3, beta=3, n_i=400, n_j=0, near=0.0, single=False,
         backward=False, diagonal=True),
    # a spin model (hard-core bosons) on a 5 x 5 lattice, an odd number of rows
    dict(name="spin_25", kind="spin", lx=5, ly=5, n_i=3001, single=False, backward=False),
    # the energy-gradient step of 28 spin orbitals: H psi from sampled onto connected configurations
    # and its backward, compensated FP32 (the benchmark's default workload)
    dict(name="step_28_f32", kind="apply", orbits=14, alpha=5, beta=5, n_i=20000, n_j=200000, near=0.0, single=True,
         backward=True, diagonal=False),
    # the same map in FP64 without a gradient, as an imaginary-time step evaluates it
    dict(name="apply_28_f64", kind="apply", orbits=14, alpha=5, beta=5, n_i=20000, n_j=200000, near=0.0, single=False,
         backward=False, diagonal=False),
    # growing the space: the 50,000 heaviest connections of those configurations
    dict(name="find_28", kind="find", orbits=14, alpha=5, beta=5, n_i=20000, near=0.0, count=50000),
    # one random neighbour per configuration (the exchange step of a sampler)
    dict(name="neighbour_28", kind="neighbour", orbits=14, alpha=5, beta=5, n_i=20000, near=0.0),
    # variational energy and its gradient over the samples of a 52-spin-orbital wave function
    dict(name="energy_52_f32", kind="energy", orbits=26, alpha=7, beta=7, n_i=65536, near=0.0, single=True),
    # the lowest eigenvector on a selected space around the reference determinant (densely connected rows)
    dict(name="lanczos_52", kind="lanczos", orbits=26, alpha=7, beta=7, n_i=16384, near=2.0, steps=12),
    # a lattice with few terms over very many rows: H psi and its backward, compensated FP32
    dict(name="hubbard_128_f32", kind="hubbard", lx=8, ly=8, alpha=32, beta=32, n_i=1000000, single=True,
         backward=True),
    # a large selected-CI growth step: the 1,000,000 heaviest connections under 3.1M terms
    dict(name="find_76", kind="find", orbits=38, alpha=10, beta=10, n_i=8192, near=0.0, count=1000000),
    # the second-order correction to a selected space
    dict(name="pt2_52", kind="pt2", orbits=26, alpha=7, beta=7, n_i=4099, near=2.0, count=200000),
    # unique configurations drawn from the autoregressive network
    dict(name="sample_52", kind="sample", sites=26, alpha=7, beta=7, hidden=512, n_i=65536),
]


def listed():
    return [dict(case) for case in _LISTED]


def _log_uniform(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    """One more case of the listed ones' ranges."""
    top = max((_cost(case) for case in _LISTED))
    while True:
        kind = rng.choice(["apply", "apply", "apply", "spin", "find", "find", "neighbour", "energy", "lanczos", "hubbard",
                           "pt2", "sample"])
        orbits = rng.randint(6, 30)
        alpha = rng.randint(2, max(2, min(10, orbits // 2)))
        beta = max(1, alpha - rng.randint(0, 1))
        space = math.comb(orbits, alpha) * math.comb(orbits, beta)
        near = rng.choice([0.0, 0.0, round(rng.uniform(1.5, 4.0), 2)])
        n_max = max(64, min(space // 4, 100000))
        n_i = min(_log_uniform(rng, 100, 65536), n_max)
        single = rng.random() < 0.5
        backward = rng.random() < 0.5
        if kind == "apply":
            n_j = rng.choice([0, min(_log_uniform(rng, 100, 200000), n_max)])
            case = dict(kind=kind, orbits=orbits, alpha=alpha, beta=beta, n_i=n_i, n_j=n_j, near=near, single=single,
                        backward=backward, diagonal=rng.random() < 0.3)
        elif kind == "spin":
            lx, ly = rng.randint(3, 6), rng.randint(3, 6)
            case = dict(kind=kind, lx=lx, ly=ly, n_i=min(_log_uniform(rng, 100, 65536), 2 ** (lx * ly) // 2),
                        single=single, backward=backward)
        elif kind == "find":
            case = dict(kind=kind, orbits=orbits, alpha=alpha, beta=beta, n_i=min(n_i, 20000), near=near,
                        count=_log_uniform(rng, 100, 300000))
        elif kind == "neighbour":
            case = dict(kind=kind, orbits=orbits, alpha=alpha, beta=beta, n_i=n_i, near=near)
        elif kind == "energy":
            case = dict(kind=kind, orbits=orbits, alpha=alpha, beta=beta, n_i=n_i, near=near, single=single)
        elif kind == "lanczos":
            case = dict(kind=kind, orbits=orbits, alpha=alpha, beta=beta, n_i=min(n_i, 16384), near=near,
                        steps=rng.randint(5, 12))
        elif kind == "hubbard":
            lx, ly = rng.randint(2, 8), rng.randint(4, 8)
            alpha, beta = lx * ly // 2, lx * ly // 2 - rng.randint(0, 1)
            n_max = math.comb(lx * ly, alpha) * math.comb(lx * ly, beta) // 4
            case = dict(kind=kind, lx=lx, ly=ly, alpha=alpha, beta=beta, n_i=min(_log_uniform(rng, 300, 1000000), n_max),
                        single=single, backward=backward)
        elif kind == "pt2":
            case = dict(kind=kind, orbits=orbits, alpha=alpha, beta=beta, n_i=min(n_i, 4099), near=near,
                        count=_log_uniform(rng, 300, 200000))
        else:
            sites = rng.randint(6, 26)
            alpha = rng.randint(2, max(2, min(7, sites // 2)))
            space = math.comb(sites, alpha) ** 2
            case = dict(kind=kind, sites=sites, alpha=alpha, beta=alpha, hidden=rng.choice([64, 128, 512]),
                        n_i=max(64, min(_log_uniform(rng, 300, 65536), space // 2)))
        # rows around the reference determinant: few out of a large space
        if case.get("near") and max(case["n_i"], case.get("n_j", 0)) > min(space // 40, 30000):
            continue
        if _cost(case) <= top:
            return case


# ---------------------------------------------------------------------------
# what a program has in hand
# ---------------------------------------------------------------------------

_MOLECULE_SEED = 2024


@functools.lru_cache(maxsize=None)
def _molecule(orbits):
    return qmb.terms.integral_hamiltonian_tables(orbits, seed=_MOLECULE_SEED)


@functools.lru_cache(maxsize=None)
def _lattice(lx, ly):
    return qmb.terms.sort_terms(*qmb.terms.prepare(qmb.terms.hubbard_dict(lx, ly, 1.0, 4.0)))


@functools.lru_cache(maxsize=None)
def _spins(lx, ly):
    """Transverse-field Ising with exchange: X on every site, ZZ and XX on every bond of the open lattice."""
    out = {}

    def add(key, value):
        out[key] = out.get(key, 0.0) + value

    for i in range(lx):
        for j in range(ly):
            a = i + j * lx
            add(((a, 1),), -0.7)
            add(((a, 0),), -0.7)
            for b in ([a + 1] if i + 1 < lx else []) + ([a + lx] if j + 1 < ly else []):
                # Z_a Z_b with Z = 1 - 2 n
                add((), 1.0)
                add(((a, 1), (a, 0)), -2.0)
                add(((b, 1), (b, 0)), -2.0)
                add(((a, 1), (a, 0), (b, 1), (b, 0)), 4.0)
                for ka in (0, 1):
                    for kb in (0, 1):
                        add(((a, ka), (b, kb)), 0.3)
    return qmb.terms.sort_terms(*qmb.terms.prepare(out))


def _tables(case):
    if case["kind"] == "spin":
        return _spins(case["lx"], case["ly"]), "bose2"
    if case["kind"] == "hubbard":
        return _lattice(case["lx"], case["ly"]), "fermi"
    return _molecule(case["orbits"]), "fermi"


@functools.lru_cache(maxsize=None)
def _hamiltonian(kind, *size):
    tables, particles = {"spin": lambda: (_spins(*size), "bose2"), "hubbard": lambda: (_lattice(*size), "fermi"),
                         "molecule": lambda: (_molecule(*size), "fermi")}[kind]()
    return qmb.Hamiltonian(tables, kind=particles)


def _handle(case):
    if case["kind"] in ("spin", "hubbard"):
        return _hamiltonian(case["kind"], case["lx"], case["ly"])
    return _hamiltonian("molecule", case["orbits"])


def _generator(seed, stream):
    return torch.Generator(device="cuda").manual_seed((int(seed) * 1000003 + stream) % (2**62))


def _pick(n, sites, filled, near, gen):
    """[n, sites] occupations with `filled` particles; near > 0: thermally spread around the lowest sites."""
    noise = torch.rand((n, sites), generator=gen, device="cuda")
    if near > 0:
        level = torch.arange(sites, device="cuda", dtype=torch.float32)
        noise = level - near * torch.log(-torch.log(noise.clamp(1e-9, 1 - 1e-7)))
    chosen = torch.argsort(noise, dim=1)[:, :filled]
    bits = torch.zeros((n, sites), dtype=torch.uint8, device="cuda")
    return bits.scatter_(1, chosen, 1)


def _pack(bits):
    n, sites = bits.shape
    nq = (sites + 7) // 8
    full = torch.zeros((n, nq * 8), dtype=torch.uint8, device=bits.device)
    full[:, :sites] = bits
    weight = (2 ** torch.arange(8, device=bits.device)).to(torch.uint8)
    return (full.view(n, nq, 8) * weight).sum(dim=2).to(torch.uint8)


def _rows(count, make, gen):
    """`count` distinct rows in lexicographic order, out of make(n)'s rows."""
    have = torch.unique(make(count + count // 8 + 64), dim=0)
    while have.shape[0] < count:
        have = torch.unique(torch.cat([have, make(2 * count + 64)]), dim=0)
    keep = torch.randperm(have.shape[0], generator=gen, device="cuda")[:count]
    return have[keep.sort().values].contiguous()


def _determinants(sites, alpha, beta, count, near, gen):
    if count >= math.comb(sites, alpha) * math.comb(sites, beta):
        return torch.from_numpy(qmb.terms.all_determinants(sites, alpha, beta)).cuda()

    spread = near

    def make(n):
        # rows around the reference determinant run out: every call spreads them a little further
        nonlocal spread
        bits = torch.empty((n, 2 * sites), dtype=torch.uint8, device="cuda")
        bits[:, 0::2] = _pick(n, sites, alpha, spread, gen)
        bits[:, 1::2] = _pick(n, sites, beta, spread, gen)
        spread *= 1.25
        return _pack(bits)

    return _rows(count, make, gen)


def _amplitudes(n, single, gen):
    pair = torch.randn((n, 2), generator=gen, device="cuda", dtype=torch.float32 if single else torch.float64)
    return torch.view_as_complex(pair)


def _inputs(case, seed):
    """The tensors a call on this case takes."""
    gen = _generator(seed, 1)
    kind = case["kind"]
    single = case.get("single", False)
    if kind == "sample":
        # the random numbers of a replayed draw, and where the program collects the configurations
        return {"uniforms": [torch.rand((case["n_i"], 4), generator=gen, device="cuda") for _ in range(case["sites"])],
                "pool": torch.zeros((case["n_i"], (2 * case["sites"] + 7) // 8), dtype=torch.uint8, device="cuda"),
                "psi": torch.zeros(case["n_i"], dtype=torch.complex128, device="cuda")}
    if kind == "spin":
        sites = case["lx"] * case["ly"]
        rows = _rows(case["n_i"], lambda n: _pack((torch.rand((n, sites), generator=gen, device="cuda") < 0.5)
                                                  .to(torch.uint8)), gen)
    elif kind == "hubbard":
        rows = _determinants(case["lx"] * case["ly"], case["alpha"], case["beta"], case["n_i"], 0.0, gen)
    else:
        rows = _determinants(case["orbits"], case["alpha"], case["beta"], case["n_i"], case["near"], gen)
    out = {"rows": rows, "psi": _amplitudes(rows.shape[0], single, gen)}
    out["targets"] = rows
    if case.get("n_j"):
        out["targets"] = _determinants(case["orbits"], case["alpha"], case["beta"], case["n_j"], case["near"], gen)
    if case.get("backward"):
        out["grad"] = _amplitudes(out["targets"].shape[0], single, gen)
    if kind == "find":
        # where the program collects the rows it finds
        out["pool"] = torch.zeros((case["count"], rows.shape[1]), dtype=torch.uint8, device="cuda")
    if kind == "neighbour":
        out["seed"] = int(torch.randint(0, 2**62, (), generator=gen, device="cuda"))
    return out


def _facing(vector, start):
    """An eigenvector's sign is free: the one that overlaps the start vector positively."""
    return vector * torch.sign(torch.vdot(start, vector).real)


def prepare(case, seed):
    state = {"case": dict(case), **_inputs(case, seed)}
    if case["kind"] == "sample":
        with torch.random.fork_rng(devices=["cuda"]):
            torch.manual_seed(int(seed))
            net = qmb.sampler.WaveFunctionElectronUpDown(
                double_sites=2 * case["sites"], physical_dim=2, is_complex=True, spin_up=case["alpha"],
                spin_down=case["beta"], hidden_size=(case["hidden"], case["hidden"]), ordering=1)
        state["net"] = net.cuda()
        return state
    state["ham"] = _handle(case)
    if case.get("backward") or case["kind"] == "energy":
        state["psi"].requires_grad_(True)
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "sample":
        configs, psi, _, _ = state["net"].generate_unique(case["n_i"], uniforms=state["uniforms"])
        for pool, part in ((state["pool"], configs), (state["psi"], psi)):
            pool[part.shape[0]:].zero_()
            pool[:part.shape[0]] = part
        return {"count": configs.shape[0], "configs": state["pool"], "psi": state["psi"]}
    ham, rows, psi, targets = state["ham"], state["rows"], state["psi"], state["targets"]
    if kind in ("apply", "spin", "hubbard"):
        out = {"hpsi": ham.apply_within(rows, psi, targets)}
        if case["backward"]:
            (out["grad"],) = torch.autograd.grad(out["hpsi"], psi, grad_outputs=state["grad"])
            out["hpsi"] = out["hpsi"].detach()
        if case.get("diagonal"):
            out["diagonal"] = ham.diagonal_term(targets)
        return out
    if kind == "find":
        found = ham.find_relative(rows, psi, case["count"])
        state["pool"][found.shape[0]:].zero_()
        state["pool"][:found.shape[0]] = found
        return {"count": found.shape[0], "rows": state["pool"]}
    if kind == "neighbour":
        return {"rows": ham.single_relative_seeded(rows, state["seed"])}
    if kind == "energy":
        energy = qmb.variational_energy(ham, rows, psi)
        (grad,) = torch.autograd.grad(energy, psi)
        return {"energy": energy.detach(), "grad": grad}
    if kind == "lanczos":
        energy, vector = qmb.lanczos_energy(ham, rows, case["steps"], start=psi)
        return {"energy": energy, "vector": _facing(vector, psi)}
    energy, correction = qmb.pt2_energy(ham, rows, psi, case["count"])
    return {"energy": energy, "correction": correction}


# ---------------------------------------------------------------------------
# the work a pass cannot do without
# ---------------------------------------------------------------------------


def _space(case):
    """(sites, terms, determinants in the space, rows one row is connected to)."""
    kind = case["kind"]
    if kind == "spin":
        sites = case["lx"] * case["ly"]
        bonds = case["lx"] * (case["ly"] - 1) + case["ly"] * (case["lx"] - 1)
        return sites, 7 * sites + 5 * bonds, 2.0**sites, sites + bonds
    if kind == "hubbard":
        n = case["lx"] * case["ly"]
        bonds = case["lx"] * (case["ly"] - 1) + case["ly"] * (case["lx"] - 1)
        return 2 * n, n + 4 * bonds, float(math.comb(n, case["alpha"])) * math.comb(n, case["beta"]), bonds
    n, a, b = case["orbits"], case["alpha"], case["beta"]
    s_a, s_b = a * (n - a), b * (n - b)
    doubles = math.comb(a, 2) * math.comb(n - a, 2) + math.comb(b, 2) * math.comb(n - b, 2) + s_a * s_b
    return 2 * n, qmb.terms.n_integral_terms(n), float(math.comb(n, a)) * math.comb(n, b), s_a + s_b + doubles


def work(case):
    kind = case["kind"]
    if kind == "sample":
        sites, n, h = case["sites"], case["n_i"], case["hidden"]
        weights = sum((2 * i) * h + h * h + 4 * h for i in range(sites)) + 2 * sites * h + h * h + h
        return {"bytes": 4 * weights + 16 * sites * n + n * ((2 * sites + 7) // 8 + 16), "flops": 2 * n * weights}
    sites, n_terms, space, connected = _space(case)
    nq = (sites + 7) // 8
    n_i = case["n_i"]
    amp = 8 if case.get("single") else 16
    table = n_terms * 28  # four (site, kind) slots and a complex coefficient
    if kind == "neighbour":
        return {"bytes": table + 2 * n_i * nq, "flops": 2 * n_terms}
    if kind == "find":
        return {"bytes": table + n_i * (nq + amp) + case["count"] * nq, "flops": 4 * n_i * connected}
    if kind == "pt2":
        return {"bytes": table + n_i * (nq + amp), "flops": 4 * n_i * connected + 8 * case["count"]}
    n_j = case.get("n_j") or n_i
    # rows reached inside the target set; clustered rows reach more (not counted)
    hits = n_i * (1 + connected * min(1.0, n_j / space))
    rows = n_i * nq + (n_j * nq if case.get("n_j") else 0)
    if kind == "energy":
        return {"bytes": table + rows + 2 * n_i * amp, "flops": 8 * hits}
    if kind == "lanczos":
        return {"bytes": table + rows + 2 * n_i * amp, "flops": 8 * hits * (case["steps"] + 2)}
    passes = 2 if case["backward"] else 1
    extra = 16 * n_j if case.get("diagonal") else 0
    return {"bytes": table + rows + passes * (n_i + n_j) * amp + extra, "flops": 8 * hits * passes}


def _cost(case):
    amount = work(case)
    return amount["bytes"] / 6.8e12 + amount["flops"] / 4e13


# ---------------------------------------------------------------------------
# the same in 64 bits, from the operators' definition
# ---------------------------------------------------------------------------


def _parity(x):
    for shift in (32, 16, 8, 4, 2, 1):
        x = x ^ (x >> shift)
    return x & 1


def _masks(site, kind, fermi, words):
    """Per term and word: sites tested, their required values, sites flipped, sites whose parity signs it."""
    site, kind = site.numpy().astype(np.int64), kind.numpy()
    n = site.shape[0]
    every = np.arange(n)
    zeros = lambda: np.zeros((n, words), dtype=np.uint64)
    mask, value, flip, par, now = zeros(), zeros(), zeros(), zeros(), zeros()
    const = np.zeros(n, dtype=np.uint64)
    live = np.ones(n, dtype=bool)
    for slot in (3, 2, 1, 0):  # the rightmost operator acts first
        on = kind[:, slot] != 2
        s = site[:, slot]
        word, bit = s // 64, np.uint64(1) << (s % 64).astype(np.uint64)
        bit = np.where(on, bit, np.uint64(0))
        create = kind[:, slot] == 1
        fresh = on & ((mask[every, word] & bit) == 0)
        mask[every, word] |= bit
        need = np.where(fresh & ~create, bit, np.uint64(0))
        value[every, word] |= need
        now[every, word] |= need
        filled = (now[every, word] & bit) != 0
        live &= ~on | (filled != create)
        if fermi:
            for w in range(words):
                span = np.clip(s - 64 * w, 0, 64)
                below = np.where(span >= 64, np.uint64(2**64 - 1),
                                 (np.uint64(1) << np.minimum(span, 63).astype(np.uint64)) - np.uint64(1))
                below = np.where(on, below, np.uint64(0))
                # the sign of the row as the earlier operators left it
                const ^= _parity((flip[:, w] & below).astype(np.uint64))
                par[:, w] ^= below
        now[every, word] ^= bit
        flip[every, word] ^= bit
    wrap = lambda a: torch.from_numpy(np.ascontiguousarray(a[live]).view(np.int64)).cuda()
    sign = torch.from_numpy(1.0 - 2.0 * const[live].astype(np.float64)).cuda()
    return wrap(mask), wrap(value), wrap(flip), wrap(par), sign, torch.from_numpy(np.nonzero(live)[0]).cuda()


def _words(rows):
    n, nq = rows.shape
    words = (nq + 7) // 8
    full = torch.zeros((n, 8 * words), dtype=torch.uint8, device=rows.device)
    full[:, :nq] = rows
    return full.view(torch.int64)


def _mixed(words):
    h = torch.zeros_like(words[:, 0])
    for q in range(words.shape[1]):
        h = (h ^ words[:, q]) * -7046029254386353131
        h = h ^ ((h >> 29) & 0x7FFFFFFFF)
    return h


class _Lookup:
    """Positions of rows in a set of rows (-1: absent)."""

    def __init__(self, words):
        self.hash, self.order = torch.sort(_mixed(words))
        self.words = words

    def __call__(self, words):
        at = torch.searchsorted(self.hash, _mixed(words)).clamp_(max=self.hash.shape[0] - 1)
        at = self.order[at]
        return torch.where((self.words[at] == words).all(dim=1), at, torch.full_like(at, -1))


def _connections(tables, fermi, words):
    """Chunks of (term, row index, image words, sign times coefficient) of every term on every row."""
    site, kind, coef = tables
    mask, value, flip, par, sign, index = _masks(site, kind, fermi, words.shape[1])
    coef = torch.view_as_complex(coef.to(torch.float64).contiguous()).cuda()[index] * sign
    step = max(1, (1 << 25) // max(1, words.shape[0]))
    for first in range(0, mask.shape[0], step):
        part = slice(first, first + step)
        bad = (words[:, None, 0] ^ value[None, part, 0]) & mask[None, part, 0]
        for q in range(1, words.shape[1]):
            bad |= (words[:, None, q] ^ value[None, part, q]) & mask[None, part, q]
        row, term = torch.nonzero(bad == 0, as_tuple=True)
        term = term + first
        image = words[row] ^ flip[term]
        odd = torch.zeros_like(row)
        for q in range(words.shape[1]):
            odd = odd ^ _parity(words[row, q] & par[term, q])
        yield term, row, image, coef[term] * (1.0 - 2.0 * odd.to(torch.float64))


def _add(out, index, value):
    torch.view_as_real(out).index_add_(0, index, torch.view_as_real(value))


def _elements(tables, fermi, rows, targets):
    """Chunks of (row index, target index, matrix element <target|H|row>)."""
    words, find = _words(rows), _Lookup(_words(targets))
    for _, row, image, value in _connections(tables, fermi, words):
        at = find(image)
        hit = at >= 0
        yield row[hit], at[hit], value[hit]


def _apply(tables, fermi, rows, psi, targets, grad=None):
    psi = psi.detach().to(torch.complex128)
    out = torch.zeros(targets.shape[0], dtype=torch.complex128, device="cuda")
    back = torch.zeros_like(psi)
    for row, at, value in _elements(tables, fermi, rows, targets):
        _add(out, at, value * psi[row])
        if grad is not None:
            _add(back, row, value.conj() * grad.to(torch.complex128)[at])
    return out, back


def _pairs(case):
    """(row, term) pairs the 64-bit computation tests."""
    return float(case["n_i"]) * _space(case)[1]


def _diagonal(tables, fermi, rows):
    words = _words(rows)
    out = torch.zeros(rows.shape[0], dtype=torch.complex128, device="cuda")
    for _, row, image, value in _connections(tables, fermi, words):
        same = (image == words[row]).all(dim=1)
        _add(out, row[same], value[same])
    return out


def _exact_lanczos(tables, rows, start, steps):
    n = rows.shape[0]
    parts = list(_elements(tables, True, rows, rows))
    row, at, value = (torch.cat([p[k] for p in parts]) for k in range(3))

    def product(x):
        y = torch.zeros(n, dtype=torch.complex128, device="cuda")
        _add(y, at, value * x[row])
        return y

    basis = [start / torch.linalg.norm(start)]
    alpha, beta = [], []
    w = product(basis[-1])
    alpha.append(torch.vdot(w, basis[-1]).real)
    w = w - alpha[-1] * basis[-1]
    for _ in range(steps + 1):
        beta.append(torch.linalg.norm(w))
        if beta[-1] < 1e-12:
            beta.pop()
            break
        basis.append(w / beta[-1])
        w = product(basis[-1])
        alpha.append(torch.vdot(w, basis[-1]).real)
        w = w - alpha[-1] * basis[-1] - beta[-1] * basis[-2]
    matrix = torch.diag(torch.stack(alpha)) + torch.diag(torch.stack(beta), 1) + torch.diag(torch.stack(beta), -1)
    values, vectors = np.linalg.eigh(matrix.cpu().numpy())
    vector = sum(float(c) * b for c, b in zip(vectors[:, 0], basis))
    return float(values[0]), vector


def _exact_pt2(tables, rows, psi, count):
    words = _words(rows)
    known = _Lookup(words)
    norm = (psi.conj() * psi).real.sum()
    hpsi, _ = _apply(tables, True, rows, psi, rows)
    energy = ((psi.conj() * hpsi).sum().real / norm).item()
    # the heaviest records outside the rows, kept in descending order chunk by chunk
    heavy = torch.empty(0, dtype=torch.float64, device="cuda")
    images = torch.empty((0, words.shape[1]), dtype=torch.int64, device="cuda")
    least = 0.0
    for _, row, image, value in _connections(tables, True, words):
        part = value * psi[row]
        weight = part.real**2 + part.imag**2
        keep = weight > least
        weight, image = weight[keep], image[keep]
        keep = known(image) < 0
        heavy, images = torch.cat([heavy, weight[keep]]), torch.cat([images, image[keep]])
        if heavy.shape[0] > 2 * count + 100000:
            heavy, at = torch.topk(heavy, count)
            images, least = images[at], float(heavy[-1])
    if heavy.shape[0] > count:
        heavy, at = torch.topk(heavy, count)
        images = images[at]
    images = torch.unique(images, dim=0)
    other = images.view(torch.uint8).view(images.shape[0], -1)[:, :rows.shape[1]].contiguous()
    if other.shape[0] == 0:
        return energy, 0.0
    hpsi, _ = _apply(tables, True, rows, psi, other)
    gap = energy - _diagonal(_flat(tables), True, other).real
    return energy, ((hpsi.real**2 + hpsi.imag**2) / norm / gap).sum().item()


def _flat(tables):
    """The terms that leave every configuration as it is."""
    site, kind, coef = tables
    _, _, flip, _, _, index = _masks(site, kind, True, (int(site.max()) + 64) // 64)
    flat = index[(flip == 0).all(dim=1)].cpu()
    return site[flat], kind[flat], coef[flat]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("find", "neighbour", "sample"):
        return None  # rows: bytes, which stay equal
    if _pairs(case) > 1.2e11:
        return None
    state = _inputs(case, seed)
    tables, particles = _tables(case)
    fermi = particles == "fermi"
    rows, psi = state["rows"], state["psi"].to(torch.complex128)
    if kind in ("apply", "spin", "hubbard"):
        hpsi, grad = _apply(tables, fermi, rows, psi, state["targets"], state.get("grad"))
        out = {"hpsi": hpsi}
        if case["backward"]:
            out["grad"] = grad
        if case.get("diagonal"):
            out["diagonal"] = _diagonal(_flat(tables), fermi, state["targets"])
        return out
    if kind == "energy":
        hpsi, _ = _apply(tables, fermi, rows, psi, rows)
        norm = (psi.conj() * psi).real.sum()
        energy = (psi.conj() * hpsi).sum().real / norm
        return {"energy": energy, "grad": 2 * (hpsi - energy * psi) / norm}
    if kind == "lanczos":
        energy, vector = _exact_lanczos(tables, rows, psi, case["steps"])
        return {"energy": energy, "vector": _facing(vector, psi)}
    energy, correction = _exact_pt2(tables, rows, psi, case["count"])
    return {"energy": energy, "correction": correction}
