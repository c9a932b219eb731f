"""The work that programs give this framework, as cases that can be timed and checked.

Every case is one pass of a program around DBSR_MAT3's or DBSR_HF's matrix set-up through the
public interface (``dbsr_gb300.Assembler``, ``gen_batch``): inputs seeded synthetic data of
``dbsr_gb300.synth`` in the shapes of its workloads.  ``kind`` says which program it is:

assemble   one partial wave: the matrix zeroed, the tables of the wave's grid built, every
           coefficient list through ``gen_matrix``, the matrix and the asymptotic
           coefficients read.  ``form`` is the precision form, ``lists`` where the caller
           holds the lists (host arrays, as a Fortran caller does, or device tensors with
           the asynchronous mode, as the assembly benchmark does), ``out`` where the matrix
           goes.
replay     the same lists again from new orbitals: the captured assembly.
batch      several independent partial waves at once (``gen_batch``).
structures one wave with every list kind Gen_matrix dispatches, perturbers and targets.
energy     E = sum c R^k(a,b;c,d) over bound orbitals and dE/dpq.
scf        the potential matrices of all orbitals of one SCF iteration (hf_matrix).
writeout   the orthogonality projection and the channel basis of an assembled matrix.

The eigensolver of the channel problems (``diag_channels``) is one library call per channel and
is not among them.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from dbsr_gb300 import FACTOR_FP64, PLAIN_FP64, SPLIT_BF16, Assembler, synth
from dbsr_gb300.api import HostMatrix, gen_batch

FORMS = {"split": SPLIT_BF16, "factor": FACTOR_FP64, "plain": PLAIN_FP64}
KS, KSP, KSQ = 9, 8, 9  # spline orders of every workload of synth
IBO = synth.IBO


# -- the cases ------------------------------------------------------------------------------------
def _assemble(form, ns, nch, mk, norb, per_slot, occupancy, z, rmax, breit=True, lists="device",
              out="device"):
    return {"kind": "assemble", "form": form, "ns": ns, "nch": nch, "mk": mk, "norb": norb,
            "per_slot": per_slot, "occupancy": occupancy, "z": z, "rmax": rmax, "breit": breit,
            "lists": lists, "out": out}


def listed():
    return [
        # the 80-spline, 2-channel wave of the smoke test and the examples: a first run, a
        # unit test, a light ion; every launch and every wait of a call counts
        dict(_assemble("split", 80, 2, 3, 4, 5, 1.0, 10.0, 25.0, breit=False, lists="host",
                       out="host"), name="wave-ns80-2ch"),
        # a middle block of the batched workload (ns 150..450, 10..300 channels, k = 0..8),
        # with an odd spline count
        dict(_assemble("split", 283, 32, 8, 20, 400, 0.05, 26.0, 40.0), name="wave-ns283-32ch"),
        # the headline shape (ns 400, k = 0..10, 20 target orbitals, 5% of the slots with 500
        # entries each, Breit) at 80 of its 120 channels, so that three matrices and their copies fit the card
        dict(_assemble("split", 400, 80, 10, 20, 500, 0.05, 26.0, 40.0), name="wave-ns400-80ch"),
        # the all-FP64 form of the factored contraction, for programs that need 1e-12
        dict(_assemble("factor", 222, 14, 6, 16, 150, 0.2, 26.0, 30.0), name="wave-fp64-ns222-14ch"),
        # the library's default form, the reference's loops on whole tables: the check run
        # that a program makes before it trusts another form
        dict(_assemble("plain", 101, 5, 3, 6, 20, 0.5, 18.0, 25.0, lists="host", out="host"),
             name="wave-plain-ns101-5ch"),
        # lists from host memory and the matrix into page-locked host memory, as a Fortran
        # caller that goes on with the matrix on the CPU has it
        dict(_assemble("split", 351, 24, 8, 20, 300, 0.1, 26.0, 40.0, lists="host",
                       out="host-window"), name="wave-to-host-ns351-24ch"),
        # relaxation cycles: the same lists from new orbitals, one graph launch a pass
        dict({k: v for k, v in _assemble("split", 200, 12, 6, 12, 100, 0.2, 26.0, 30.0).items()
              if k not in ("lists", "out")}, kind="replay", name="replay-ns200-12ch"),
        # J-parity blocks of different sizes built side by side
        {"name": "batch-4-waves", "kind": "batch", "nwaves": 4, "ns": 150, "ns_step": 41, "nch": 10,
         "mk": 8, "norb": 20, "per_slot": 300, "occupancy": 0.1, "z": 26.0, "rmax": 40.0},
        # every list kind of a real bank: bound-bound, bound-channel and channel-channel
        # integrals, overlaps, one-electron lists, perturbers, targets
        {"name": "structures-ns180-6ch", "kind": "structures", "ns": 180, "nch": 6, "mk": 3,
         "norb": 10, "npert": 4, "ntarg": 3, "per_list": 200, "n_entries": 6000, "z": 18.0,
         "rmax": 25.0},
        # the differentiation workload: ns 300, 30 orbitals, k = 0..8, 5e4 entries
        {"name": "energy-ns300-30orb", "kind": "energy", "ns": 300, "norb": 30, "kmax": 8,
         "n_entries": 50000, "z": 18.0, "rmax": 30.0},
        # one SCF iteration over the same basis
        {"name": "scf-ns300-30orb", "kind": "scf", "ns": 300, "norb": 30, "kmax": 8, "z": 18.0,
         "rmax": 30.0, "form": "split"},
        # what follows an assembly before the matrix is recorded
        {"name": "writeout-ns250-16ch", "kind": "writeout", "ns": 250, "nch": 16, "norb": 12,
         "z": 26.0, "rmax": 30.0, "form": "split"},
    ]


def draw(rng):
    """One more case: ns 60..400, 2..80 channels, the multipoles, orbital counts and entry counts
    of the listed ones."""

    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["assemble"] * 5 + ["replay", "batch", "structures", "energy", "scf",
                                          "writeout"])
    z, rmax = float(rng.choice([10.0, 18.0, 26.0])), float(rng.randint(20, 40))
    if kind in ("assemble", "replay"):
        form = rng.choice(["split"] * 4 + ["factor", "plain"]) if kind == "assemble" else "split"
        # the whole tables of the plain form and its loops bound its sizes
        ns = {"split": log(60, 400), "factor": log(60, 250), "plain": log(60, 110)}[form]
        nch = {"split": log(2, 64), "factor": log(2, 16), "plain": log(2, 5)}[form]
        mk = rng.randint(2, 10 if form == "split" else 4)
        c = _assemble(form, ns, min(nch, 24) if kind == "replay" else nch, mk, rng.randint(4, 20),
                      log(5, 500), 0.05 if nch > 24 else rng.choice([0.1, 0.2, 0.5]), z, rmax,
                      breit=rng.random() < 0.7,
                      lists=rng.choice(["device", "host"]),
                      out=rng.choice(["device", "device", "host-window" if form == "split" else "device"]))
        if kind == "replay":
            c = dict({k: v for k, v in c.items() if k not in ("lists", "out")}, kind="replay")
        return c
    if kind == "batch":
        return {"kind": "batch", "nwaves": rng.randint(2, 6), "ns": rng.randint(70, 200),
                "ns_step": rng.randint(5, 35), "nch": log(3, 14), "mk": rng.randint(2, 8),
                "norb": rng.randint(4, 20), "per_slot": log(5, 400), "occupancy": 0.1, "z": z,
                "rmax": rmax}
    if kind == "structures":
        return {"kind": "structures", "ns": log(60, 220), "nch": rng.randint(2, 8),
                "mk": rng.randint(1, 4), "norb": rng.randint(4, 12), "npert": rng.randint(1, 6),
                "ntarg": rng.randint(1, 3), "per_list": log(20, 300), "n_entries": log(300, 8000),
                "z": z, "rmax": rmax}
    if kind == "energy":
        return {"kind": "energy", "ns": log(60, 300), "norb": rng.randint(4, 30),
                "kmax": rng.randint(2, 8), "n_entries": log(200, 50000), "z": z, "rmax": rmax}
    if kind == "scf":
        return {"kind": "scf", "ns": log(60, 300), "norb": rng.randint(4, 30),
                "kmax": rng.randint(2, 8), "z": z, "rmax": rmax, "form": "split"}
    return {"kind": "writeout", "ns": log(60, 300), "nch": rng.randint(2, 16),
            "norb": rng.randint(4, 14), "z": z, "rmax": rmax, "form": "split"}


# -- inputs ---------------------------------------------------------------------------------------
def _rmax(case):
    # at least ten geometric intervals below r = 1, as in synth's reduced workloads
    return min(case["rmax"], 1.0 + 0.5 * ((case["ns"] - KS + 1) - 11))


def _workload(case, seed):
    """A wave in the shape of synth's workloads: ``per_slot`` entries in ``occupancy`` of the
    (channel pair, k) slots, and one overlap entry per channel pair on average."""
    nch, mk = case["nch"], case["mk"]
    slots = max(1, int(round(case["occupancy"] * (nch * (nch + 1) // 2) * (mk + 1))))
    w = synth.small(ns=case["ns"], nch=nch, mk=mk, n_entries=case["per_slot"] * slots,
                    breit=case.get("breit", True), seed=seed, rmax=case["rmax"], z=case["z"],
                    occupancy=case["occupancy"], norb=case["norb"])
    rng = np.random.Generator(np.random.Philox(seed + 31))
    n, nb = 4 * nch, w.nbound
    k1 = (nb + rng.integers(1, nch + 1, n)) * IBO + rng.integers(1, nb + 1, n)
    k2 = (nb + rng.integers(1, nch + 1, n)) * IBO + rng.integers(1, nb + 1, n)
    zero = np.zeros(n, dtype=np.int64)
    w.lists = [L for L in w.lists if L.icase != 0]
    w.lists.insert(0, synth.CList(0, 3, 0, *synth.sort_merge(k1, k2, zero, zero,
                                                             rng.uniform(-1.0, 1.0, n))))
    return w


def _lists(w, where):
    out = []
    for L in w.lists:
        a = [L.k1, L.k2, L.k3, L.k4, L.c]
        if where == "device":
            a = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in a]
        out.append((L.icase, L.itype, L.kpol, *a))
    return out


def _assembler(w, form):
    a = Assembler(w.t, w.ks, w.ksp, w.ksq)
    a.set_orbitals(w.pq, w.ipbs)
    a.alloc_matrix(w.nch, w.icc, w.iicc, w.mk)
    a.set_precision(FORMS[form])
    return a


class _Device:
    """hch(ms,ms,iicc) where the library holds it, for torch: (block, column, row).  Holds the
    assembler, so that the memory lives as long as a tensor over it."""

    def __init__(self, a):
        self.assembler = a
        self.__cuda_array_interface__ = {"data": (a.matrix_device_ptr(), False), "version": 3,
                                         "shape": (a.iicc, a.ms, a.ms), "typestr": "<f8",
                                         "strides": None}


class _Host:
    """The array of a HostMatrix, holding it likewise."""

    def __init__(self, n):
        self.matrix = HostMatrix(n)
        self.__array_interface__ = self.matrix.array.__array_interface__


def _matrix_view(a):
    return torch.as_tensor(_Device(a), device="cuda")


def _scf_coefficients(case, seed):
    """a(i,j,k) and b(i,j,k) of an energy expression where its selection rules allow them."""
    norb, kmax = case["norb"], case["kmax"]
    kap = [k for _, k in synth.TARGET_ORBITALS[:norb]]
    ls, j2 = [synth.l_kappa(k) for k in kap], [synth.j2_kappa(k) for k in kap]
    coef = np.random.Generator(np.random.Philox(seed + 5)).uniform(-1.0, 1.0, (norb, norb, kmax + 1))
    A, B = np.zeros_like(coef), np.zeros_like(coef)
    for i in range(norb):
        for j in range(norb):
            for k in range(kmax + 1):
                if k % 2 == 0 and k <= (j2[i] + j2[j]) // 2:
                    A[i, j, k] = coef[max(i, j), min(i, j), k]
                if i != j and (k + ls[i] + ls[j]) % 2 == 0 and \
                        abs(j2[i] - j2[j]) // 2 <= k <= (j2[i] + j2[j]) // 2:
                    B[i, j, k] = coef[min(i, j), max(i, j), k]
    return A, B


def _energy(case, seed, n=None):
    return synth.energy_workload("energy", seed, case["ns"], _rmax(case), case["z"], case["norb"],
                                 case["kmax"], n or case["n_entries"])


def _writeout(case, seed):
    """An assembled matrix and its channel solutions: blocks with the decay and the range of
    magnitudes of Hamiltonian blocks over B-splines (large near the nucleus, falling off the
    diagonal), solutions orthonormal and localised, half of them kept."""
    ns, nch = case["ns"], case["nch"]
    ms, iicc = 2 * ns, case["nch"] * (case["nch"] + 1) // 2
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = torch.arange(ms, device="cuda", dtype=torch.float64) % ns
    scale = torch.exp(-4.0 * r / ns)
    decay = torch.exp(-(r[:, None] - r[None, :]).abs() / 12.0)
    h = torch.randn(iicc, ms, ms, generator=g, device="cuda", dtype=torch.float64)
    h *= decay * (scale[:, None] * scale[None, :])
    h[:nch] = 0.5 * (h[:nch] + h[:nch].transpose(1, 2))  # the diagonal blocks come first
    m = torch.randn(min(nch, 3), ms, ms, generator=g, device="cuda", dtype=torch.float64) * decay
    q = torch.linalg.qr(m + 2.0 * torch.eye(ms, device="cuda", dtype=torch.float64))[0]
    sol = torch.stack([q[i % q.shape[0]] for i in range(nch)])  # (channel, solution, spline)
    rng = np.random.Generator(np.random.Philox(seed + 3))
    nsol = rng.integers(ms // 2 - 5, ms // 2 + 6, nch).astype(np.int32)
    for i in range(nch):
        sol[i, int(nsol[i]):] = 0.0
    nb = case["norb"]
    kb = [k for _, k in synth.TARGET_ORBITALS[:nb]]
    kc = rng.choice(sorted(set(kb)), nch)
    iort = np.zeros((nb + nch, nch), dtype=np.int32, order="F")
    for i in range(nch):
        iort[[j for j in range(nb) if kb[j] == kc[i]], i] = 1
    return h, sol.contiguous(), nsol, iort


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("assemble", "replay"):
        w = _workload(case, seed)
        a = _assembler(w, case["form"])
        s = {"a": a, "w": w, "lists": _lists(w, case.get("lists", "device")), "view": _matrix_view(a)}
        if kind == "replay":
            a.graph_capture(s["lists"])
            rng = np.random.Generator(np.random.Philox(seed + 77))
            pq = w.pq * (1.0 + rng.uniform(-1e-3, 1e-3, w.pq.shape))  # the next cycle's orbitals
            s["pq"] = torch.from_numpy(np.ascontiguousarray(pq.transpose(2, 1, 0))).cuda()
        elif case["lists"] == "device":
            a.set_async(True)
        if case.get("out") == "host-window":
            s["host"] = np.asarray(_Host(a.ms * a.ms * a.iicc))
        elif case.get("out") == "host":
            s["out"] = np.zeros((a.ms, a.ms, a.iicc), order="F")
        torch.cuda.synchronize()
        return dict(s, case=case)
    if kind == "batch":
        ws = [_workload(dict(case, ns=case["ns"] + i * case["ns_step"], nch=case["nch"] + i), seed + i)
              for i in range(case["nwaves"])]
        asm = [_assembler(w, "split") for w in ws]
        s = {"a": asm, "w": ws, "lists": [_lists(w, "device") for w in ws],
             "view": [_matrix_view(a) for a in asm], "case": case}
        torch.cuda.synchronize()
        return s
    if kind == "structures":
        kw = dict(ns=case["ns"], nch=case["nch"], mk=case["mk"], norb=case["norb"], seed=seed,
                  rmax=case["rmax"], z=case["z"])
        w = synth.structures_case(npert=case["npert"], ntarg=case["ntarg"],
                                  per_list=case["per_list"], **kw)
        w.lists = synth.small(n_entries=case["n_entries"], breit=True, **kw).lists + w.lists
        a = _assembler(w, "split")
        a.alloc_perturbers(w.npert, w.icb, w.ibb)
        a.set_targets(w.ntarg, w.iptar, w.iitar)
        a.set_dhl(w.kap_list, w.hd, w.kbs)
        return {"a": a, "w": w, "lists": _lists(w, "host"), "view": _matrix_view(a), "case": case}
    if kind == "energy":
        w = _energy(case, seed)
        a = Assembler(w.t, w.ks, w.ksp, w.ksq)
        return {"a": a, "w": w, "case": case}
    if kind == "scf":
        w = _energy(case, seed, 8)
        norb = case["norb"]
        a = Assembler(w.t, w.ks, w.ksp, w.ksq)
        a.set_orbitals(w.pq, np.zeros(norb, np.int32))
        a.alloc_matrix(1, np.ones((1, 1), np.int32, order="F"), 1, case["kmax"])
        a.set_precision(FORMS[case["form"]])
        A, B = _scf_coefficients(case, seed)
        out = torch.empty(norb, a.ms, a.ms, dtype=torch.float64, device="cuda")
        return {"a": a, "w": w, "A": A, "B": B, "out": out, "case": case}
    ns, nch, nb = case["ns"], case["nch"], case["norb"]
    t = synth.knots(ns, _rmax(case), case["z"], KS)
    rng = np.random.Generator(np.random.Philox(seed))
    pq = np.zeros((ns, 2, nb + nch), order="F")
    pq[:, :, :nb] = synth.orbital_coefficients(t, KS, KSP, KSQ, case["z"],
                                               synth.TARGET_ORBITALS[:nb], rng)
    ipbs = np.zeros(nb + nch, dtype=np.int32)
    ipbs[nb:] = np.arange(1, nch + 1)
    a = Assembler(t, KS, KSP, KSQ)
    a.set_orbitals(pq, ipbs)
    a.alloc_matrix(nch, synth.block_numbering(nch), nch * (nch + 1) // 2, 0)
    a.set_precision(FORMS[case["form"]])
    h, sol, nsol, iort = _writeout(case, seed)
    torch.cuda.synchronize()
    return {"a": a, "h": h, "sol": sol, "nsol": nsol, "iort": iort, "view": _matrix_view(a),
            "case": case, "t": t, "pq": pq}


# -- one pass -------------------------------------------------------------------------------------
def run(state):
    case, a = state["case"], state["a"]
    kind = case["kind"]
    if kind == "assemble":
        if case["out"] == "host-window":
            a.invalidate_tables()
            out, acf = a.assemble_to_host(state["lists"], out=state["host"])
            return {"hch": out, "acf": acf}
        a.zero_matrix()
        a.invalidate_tables()  # a new wave: its tables and orbital products are built
        for item in state["lists"]:
            a.gen_matrix(*item)
        if case["out"] == "host":
            return {"hch": a.get_matrix(out=state["out"]), "acf": a.get_acf()}
        a.sync()
        return {"hch": state["view"], "acf": a.get_acf()}
    if kind == "replay":
        a.graph_launch(state["pq"])
        return {"hch": state["view"], "acf": a.get_acf()}
    if kind == "batch":
        for x in a:
            x.zero_matrix()
            x.invalidate_tables()
        gen_batch(a, state["lists"])
        return {"hch": state["view"], "acf": [x.get_acf() for x in a]}
    if kind == "structures":
        a.zero_matrix()
        a.invalidate_tables()
        for item in state["lists"]:
            a.gen_matrix(*item)
        hcp, hp = a.get_perturbers()
        htarg, otarg = a.get_targets()
        return {"hch": state["view"], "acf": a.get_acf(), "hcp": hcp, "hp": hp, "htarg": htarg,
                "otarg": otarg}
    if kind == "energy":
        w = state["w"]
        a.set_orbitals(w.pq, w.ipbs)  # the orbitals of this evaluation
        e, g = a.backward(w.k, w.i1, w.i2, w.i3, w.i4, w.coef)
        return {"energy": np.float64(e), "gradient": g}
    if kind == "scf":
        # new orbitals every iteration; the tables depend on the grid only and stay
        a.set_orbitals(state["w"].pq, np.zeros(case["norb"], np.int32))
        for i in range(case["norb"]):
            a.hf_matrix(i + 1, state["A"][i], state["B"][i], 1.0, out=state["out"][i])
        return state["out"]
    state["view"].copy_(state["h"])  # the assembled matrix
    torch.cuda.current_stream().synchronize()  # the library works on a stream of its own
    a.orth_channels(state["iort"])
    orth = state["view"].clone()
    torch.cuda.current_stream().synchronize()
    a.channel_basis(state["sol"], state["nsol"])
    return {"orth": orth, "basis": state["view"]}


# -- what a pass cannot do without ----------------------------------------------------------------
def _wave_work(case):
    """Matrix written once and lists read once; a result of rank norb per exchange segment and PQ
    type, a band of entries per direct one; one segment an occupied slot and kind."""
    ns, nch, mk = case["ns"], case["nch"], case["mk"]
    pairs = nch * (nch + 1) // 2
    occ = case.get("occupancy", 1.0)
    slots = max(1.0, occ * pairs * (mk + 1))
    entries = slots * case["per_slot"] if "per_slot" in case else case["n_entries"]
    nbytes = 8.0 * pairs * 4 * ns * ns + 24.0 * entries
    if case.get("breit", True):
        results = slots * (4 + 2 * 1.0)  # R^k exchange: four types; S^k: about two lists
        direct = entries * (4 * KS + 2 * (2 * KS - 1)) / 4.0
    else:
        results, direct = slots * 4.0, entries * 4 * KS / 2.0
    return nbytes, 2.0 * ns * ns * case["norb"] * results + 2.0 * ns * direct


def work(case):
    kind = case["kind"]
    if kind in ("assemble", "replay", "structures"):
        b, f = _wave_work(case)
        return {"bytes": b, "flops": f}
    if kind == "batch":
        b = f = 0.0
        for i in range(case["nwaves"]):
            x, y = _wave_work(dict(case, ns=case["ns"] + i * case["ns_step"], nch=case["nch"] + i))
            b, f = b + x, f + y
        return {"bytes": b, "flops": f}
    ns, nb = case["ns"], case["norb"]
    if kind == "energy":
        # every pair potential of half the multipoles once (four types, a band of ns x 9, nine
        # cells a value), each entry a dot of two bands; gradients as band times vector
        pairs = nb * (nb + 1) / 2 * (case["kmax"] + 1) / 2 * 4
        return {"bytes": 8.0 * 4 * ns * nb + 28.0 * case["n_entries"],
                "flops": 2.0 * pairs * ns * KS * KS + 2.0 * case["n_entries"] * 4 * ns * KS}
    if kind == "scf":
        return {"bytes": 8.0 * nb * 4 * ns * ns,
                "flops": nb * (case["kmax"] + 1) * 4 * 2.0 * ns * ns * nb / 2}
    ms, nch = 2 * ns, case["nch"]
    blocks = nch * (nch + 1) // 2
    off = nch * (nch - 1) // 2
    return {"bytes": 8.0 * ms * ms * (3 * blocks + nch),
            "flops": off * 2.0 * (ms // 2) * (ms * ms + ms * (ms // 2)) + blocks * 8.0 * ms * ms}


# -- the same in 64 bits, from the definitions ----------------------------------------------------
class _Exact:
    """R^k and S^k contractions over cells: a table is a sum over pairs of knot intervals, a
    product of one-dimensional moments where the intervals differ and a nested Gauss sum where
    they agree.  Functions are P (0) and Q (1); arrays are FP64 on the GPU, the P basis padded to
    nine local functions."""

    def __init__(self, t, z=None):
        self.t = t
        self.ns = t.size - KS
        self.nv = self.ns - KS + 1
        x, w = np.polynomial.legendre.leggauss(KS)
        x, w = 0.5 * (x + 1.0), 0.5 * w
        lo, hi = t[KS - 1:KS - 1 + self.nv], t[KS:KS + self.nv]
        r = lo[:, None] + (hi - lo)[:, None] * x
        self.r, self.w = self._dev(r), self._dev((hi - lo)[:, None] * w)
        rin = lo[:, None, None] + (r - lo[:, None])[:, :, None] * x  # points below each r
        self.rin, self.win = self._dev(rin), self._dev((r - lo[:, None])[:, :, None] * w)
        self.f = [self._dev(self._splines(k, r)) for k in (KSP, KSQ)]
        self.fin = [self._dev(self._splines(k, rin.reshape(self.nv, -1)).reshape(
            self.nv, KS, KS, KS)) for k in (KSP, KSQ)]
        loc = torch.arange(KS, device="cuda")
        self.idx = torch.arange(self.nv, device="cuda")[:, None] + loc  # (nv, 9) function numbers

    @staticmethod
    def _dev(a):
        return torch.from_numpy(np.ascontiguousarray(a)).cuda()

    def _splines(self, k, x):
        """Values of the k splines of order k on interval v at x[v, :]: (nv, points, 9)."""
        nv = self.nv
        inner = self.t[KS - 1:KS + nv]
        tx = np.concatenate([np.full(k - 1, inner[0]), inner, np.full(k - 1, inner[-1])])
        v = np.arange(nv)
        out = np.zeros(x.shape + (KS,))
        out[..., 0] = 1.0
        for j in range(1, k):  # Cox-de Boor on one interval
            prev, out = out, np.zeros_like(out)
            for m in range(j):
                right = tx[v + k - 1 + m + 1][:, None]
                left = tx[v + k - 1 + m + 1 - j][:, None]
                q = prev[..., m] / (right - left)
                out[..., m] += (right - x) * q
                out[..., m + 1] += (x - left) * q
        return out

    def moment(self, a, b, k):
        return torch.einsum("vm,vmi,vmj->vij", self.w * self.r ** k, self.f[a], self.f[b])

    def table(self, family, typ, k):
        """(lo1, hi1, lo2, hi2, cell): the moments of both electrons' pairs and the integrals of
        the common interval (i, i', j, j'); hi1 and lo2 are None for S^k (first electron inside)."""
        if family == "R":
            e1 = (typ in (1, 3),) * 2
            e2 = (typ in (1, 2),) * 2
        else:
            e1, e2 = (0, 1), ((0, 1) if typ == 0 else (1, 0))
        e1, e2 = tuple(int(x) for x in e1), tuple(int(x) for x in e2)

        def outer(e):
            return torch.einsum("vm,vmi,vmj->vmij", self.w * self.r ** (-(k + 1)), self.f[e[0]],
                                self.f[e[1]])

        def inner(e):
            return torch.einsum("vmn,vmni,vmnj->vmij", self.win * self.rin ** k, self.fin[e[0]],
                                self.fin[e[1]])

        cell = torch.einsum("vmij,vmkl->vijkl", inner(e1), outer(e2))
        lo1, hi2 = self.moment(*e1, k), self.moment(*e2, -(k + 1))
        if family == "S":
            return lo1, None, None, hi2, cell
        cell = cell + torch.einsum("vmij,vmkl->vijkl", outer(e1), inner(e2))
        return lo1, self.moment(*e1, -(k + 1)), self.moment(*e2, k), hi2, cell

    def cells(self, p, q):
        """p(i) q(j) on every interval; p, q (..., ns)."""
        return torch.einsum("...vi,...vj->...vij", p[..., self.idx], q[..., self.idx])

    def direct(self, tab, side, d):
        """Potential on electron `side` of the density cells d (..., nv, 9, 9) of the other."""
        lo1, hi1, lo2, hi2, cell = tab

        def before(x):  # sums over earlier intervals (the terms span many decades: no difference)
            return torch.cat([torch.zeros_like(x[..., :1]), torch.cumsum(x, -1)[..., :-1]], -1)

        def after(x):
            return torch.flip(before(torch.flip(x, (-1,))), (-1,))

        def dot(m):
            return torch.einsum("vij,...vij->...v", m, d)

        if side == 1:
            v = torch.einsum("vijkl,...vkl->...vij", cell, d)
            v = v + after(dot(hi2))[..., None, None] * lo1
            if hi1 is not None:
                v = v + before(dot(lo2))[..., None, None] * hi1
        else:
            v = torch.einsum("vijkl,...vij->...vkl", cell, d)
            v = v + before(dot(lo1))[..., None, None] * hi2
            if hi1 is not None:
                v = v + after(dot(hi1))[..., None, None] * lo2
        return v

    def full(self, v):
        """(ns, ns) from cells (nv, 9, 9)."""
        out = torch.zeros(self.ns, self.ns, dtype=torch.float64, device="cuda")
        out.index_put_((self.idx[:, :, None].expand(-1, -1, KS), self.idx[:, None, :].expand(
            -1, KS, -1)), v, accumulate=True)
        return out

    def exchange(self, tab, case34, d):
        """case 3: sum d(i',j) T(i,i';j,j') as (i, j'); case 4: sum d(i,j') T as (i', j)."""
        lo1, hi1, lo2, hi2, cell = tab
        if case34 == 4:
            lo1, hi2 = lo1.transpose(1, 2), hi2.transpose(1, 2)
            if hi1 is not None:
                hi1, lo2 = hi1.transpose(1, 2), lo2.transpose(1, 2)
            cell = cell.permute(0, 2, 1, 4, 3)
        nv, ns = self.nv, self.ns

        def far(m1, m2, upper):
            x = torch.einsum("vij,vjc->vic", m1, d[self.idx])            # (nv, 9, ns)
            x = torch.einsum("viwj,wjk->viwk", x[..., self.idx], m2)     # (nv, 9, nv, 9)
            order = torch.arange(nv, device="cuda")
            keep = order[:, None] < order[None, :] if upper else order[:, None] > order[None, :]
            return (x * keep[:, None, :, None]).reshape(nv * KS, nv * KS)

        x = far(lo1, hi2, True)
        if hi1 is not None:
            x += far(hi1, lo2, False)
        flat = self.idx.reshape(-1)
        rows = torch.zeros(ns, nv * KS, dtype=torch.float64, device="cuda").index_add_(0, flat, x)
        out = torch.zeros(ns, ns, dtype=torch.float64, device="cuda").index_add_(1, flat, rows)
        near = d[self.idx[:, :, None], self.idx[:, None, :]]             # (nv, i', j)
        return out + self.full(torch.einsum("vxijy,vij->vxy", cell, near))

    def overlap(self, comp):
        return self.full(self.moment(comp, comp, 0))


R_DIRECT = ((0, 0), (1, 1), (1, 0), (0, 1))    # per type: (components of the density, quadrant)
R_EXCH = ((0, 0), (1, 1), (0, 1), (1, 0))
S_SPEC = {6: ((0, 1), (0, 1), 1), 7: ((0, 1), (0, 1), 2), 8: ((0, 1), (1, 0), 3),
          9: ((1, 0), (0, 1), 4), 16: ((0, 1), (1, 0), 1), 17: ((1, 0), (0, 1), 2),
          18: ((0, 0), (1, 1), 3), 19: ((1, 1), (0, 0), 4)}  # (quadrant, components, case)


def _exact_wave(w, pq):
    """hch (block, column, row) and acf of a wave's lists over the orbitals pq(ns,2,nbf)."""
    ex = _Exact(w.t)
    ns, ms = ex.ns, 2 * ex.ns
    orb = ex._dev(pq.transpose(2, 1, 0))  # (orbital, component, ns)
    hch = torch.zeros(w.iicc, ms, ms, dtype=torch.float64, device="cuda")  # [b][column][row]
    acf = np.zeros((w.iicc, w.mk + 1))
    grams = [ex.overlap(0), ex.overlap(1)]

    def add(ich, jch, y, quad):
        b = int(w.icc[ich - 1, jch - 1]) - 1
        r, c = slice(quad[0] * ns, quad[0] * ns + ns), slice(quad[1] * ns, quad[1] * ns + ns)
        if ich > jch:
            hch[b, c, r] += y.T
        elif ich < jch:
            hch[b, c, r] += y
        else:
            hch[b, c, r] += 0.5 * y.T
            hch[b, r, c] += 0.5 * y

    for L in w.lists:
        if L.icase == 0:
            v = torch.cat([orb[:, q] @ grams[q] for q in (0, 1)], 1)
            for i in range(L.n):
                i1, i2 = divmod(int(L.k1[i]), IBO)
                j1, j2 = divmod(int(L.k2[i]), IBO)
                ich, jch = int(w.ipbs[i1 - 1]), int(w.ipbs[j1 - 1])
                b, c = int(w.icc[ich - 1, jch - 1]) - 1, float(L.c[i])
                x = torch.outer(v[j2 - 1], v[i2 - 1])  # [column][row] of v(row) w(column)
                hch[b] += c * x if ich > jch else c * x.T if ich < jch else 0.5 * c * (x + x.T)
            continue
        cuts = np.flatnonzero(np.r_[True, L.k1[1:] != L.k1[:-1], True])
        a, b2, c = (torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (L.k2, L.k3, L.c))
        a, b2 = a.long() - 1, b2.long() - 1
        if L.icase == 2:
            todo = [("R", q, (R_DIRECT if L.itype == 3 else R_EXCH)[q], 1 if L.itype == 3 else 3)
                    for q in range(4)]
        else:
            todo = [("S", L.itype // 10, None, S_SPEC[L.itype][2])]
        for family, typ, comp, case in todo:
            tab = ex.table(family, typ, L.kpol)
            if family == "S":
                quad, (c1, c2), _ = S_SPEC[L.itype]
            elif L.itype == 3:  # density over the second electron, result on the first
                c1 = c2 = (0, 1, 1, 0)[typ]
                quad = ((0, 0), (1, 1), (0, 0), (1, 1))[typ]
            else:
                (c1, c2), quad = comp, comp
            p, q = orb[:, c1], orb[:, c2]
            acfm = grams_k = None
            if family == "R" and L.itype == 3 and typ <= 1:
                grams_k = ex.full(ex.moment(typ, typ, L.kpol))
                acfm = orb[:, typ] @ grams_k @ orb[:, typ].T
            for s in range(len(cuts) - 1):
                e = slice(int(cuts[s]), int(cuts[s + 1]))
                ich, jch = divmod(int(L.k1[cuts[s]]), IBO)
                d = (p[a[e]] * c[e, None]).T @ q[b2[e]]
                if case <= 2:
                    cell = d[ex.idx[:, :, None], ex.idx[:, None, :]]
                    y = ex.full(ex.direct(tab, case, cell))
                else:
                    y = ex.exchange(tab, case, d)
                if family == "R" and L.itype == 3:
                    y = 0.5 * (y + y.T)
                add(ich, jch, y, quad)
                if acfm is not None:
                    blk = int(w.icc[ich - 1, jch - 1]) - 1
                    acf[blk, L.kpol] += float((c[e] * acfm[a[e], b2[e]]).sum())
    return hch, acf


def _exact_energy(w):
    ex = _Exact(w.t)
    orb = ex._dev(w.pq.transpose(2, 1, 0))
    nb = orb.shape[0]
    g = torch.zeros_like(orb)
    e = torch.zeros((), dtype=torch.float64, device="cuda")
    dev = lambda x: torch.from_numpy(np.ascontiguousarray(x)).cuda()  # noqa: E731
    i1, i2, i3, i4 = (dev(x).long() - 1 for x in (w.i1, w.i2, w.i3, w.i4))
    k, coef = dev(w.k), dev(w.coef)
    for kk in range(int(w.k.max()) + 1):
        m = k == kk
        if not bool(m.any()):
            continue
        c = torch.zeros(nb * nb, nb * nb, dtype=torch.float64, device="cuda")  # (a,c) x (b,d)
        c.index_put_((i1[m] * nb + i3[m], i2[m] * nb + i4[m]), coef[m], accumulate=True)
        for typ in range(4):
            A, B = int(typ in (1, 3)), int(typ in (1, 2))
            tab = ex.table("R", typ, kk)
            for side, x, mat in ((1, B, c), (2, A, c.T)):
                y = A if side == 1 else B
                rows = torch.nonzero(mat.abs().sum(1)).reshape(-1)
                for part in torch.split(rows, 128):
                    rho = ex.cells(orb[:, None, x].expand(nb, nb, -1).reshape(nb * nb, -1),
                                   orb[None, :, x].expand(nb, nb, -1).reshape(nb * nb, -1))
                    d = (mat[part] @ rho.reshape(nb * nb, -1)).reshape(-1, ex.nv, KS, KS)
                    v = ex.direct(tab, side, 0.5 * (d + d.transpose(-1, -2)))
                    p, q = part // nb, part % nb
                    for u, f in ((p, q), (q, p)):
                        loc = torch.einsum("pvij,pvj->pvi", v, orb[f, y][:, ex.idx])
                        vec = torch.zeros(part.numel(), ex.ns, dtype=torch.float64, device="cuda")
                        vec.index_add_(1, ex.idx.reshape(-1), loc.reshape(part.numel(), -1))
                        g[:, y].index_add_(0, u, vec)
                        if side == 1 and u is p:
                            e = e + (vec * orb[p, y]).sum()
    return np.float64(float(e)), g.permute(2, 1, 0).cpu().numpy()


def _exact_scf(case, seed):
    w = _energy(case, seed, 8)
    A, B = _scf_coefficients(case, seed)
    ex = _Exact(w.t)
    ns, norb = ex.ns, case["norb"]
    orb = ex._dev(w.pq.transpose(2, 1, 0))
    out = torch.zeros(norb, 2 * ns, 2 * ns, dtype=torch.float64, device="cuda")
    for kk in range(case["kmax"] + 1):
        for ii, jj, typ in ((0, 0, 0), (0, 1, 2), (1, 0, 3), (1, 1, 1)):
            tab = ex.table("R", typ, kk)
            si, sj = slice(ii * ns, ii * ns + ns), slice(jj * ns, jj * ns + ns)
            for i in range(norb):
                a, b = A[i, :, kk].copy(), ex._dev(B[i, :, kk])
                a[i] *= 2.0
                if a.any():
                    d = (orb[:, jj] * ex._dev(a)[:, None]).T @ orb[:, jj]
                    y = ex.full(ex.direct(tab, 1, d[ex.idx[:, :, None], ex.idx[:, None, :]]))
                    out[i, si, si] += 0.5 * (y + y.T)
                if bool(b.any()):
                    y = ex.exchange(tab, 4, (orb[:, ii] * b[:, None]).T @ orb[:, jj])
                    out[i, si, sj] += 0.5 * y
                    out[i, sj, si] += 0.5 * y.T
    return out  # symmetric: the order of rows and columns does not matter


def _exact_writeout(case, seed):
    ns, nch, nb = case["ns"], case["nch"], case["norb"]
    t = synth.knots(ns, _rmax(case), case["z"], KS)
    rng = np.random.Generator(np.random.Philox(seed))
    pq = synth.orbital_coefficients(t, KS, KSP, KSQ, case["z"], synth.TARGET_ORBITALS[:nb], rng)
    ex = _Exact(t)
    orb = ex._dev(pq.transpose(2, 1, 0))
    v = torch.cat([orb[:, 0], orb[:, 1]], 1)
    u = torch.cat([orb[:, 0] @ ex.overlap(0), orb[:, 1] @ ex.overlap(1)], 1)
    h, sol, nsol, iort = _writeout(case, seed)
    icc = synth.block_numbering(nch)
    eye = torch.eye(2 * ns, dtype=torch.float64, device="cuda")
    proj = []  # 1 - sum_j w_j v_j^T
    for i in range(nch):
        on = torch.from_numpy(np.flatnonzero(iort[:nb, i])).cuda()
        proj.append(eye - u[on].T @ v[on])
    orth, basis = torch.empty_like(h), torch.empty_like(h)
    for i in range(nch):
        for j in range(i + 1):
            b = int(icc[i, j]) - 1
            x = proj[i] @ h[b].T @ proj[j].T  # rows: channel i
            orth[b] = x.T
            if i == j:
                basis[b] = x.T
                continue
            y = torch.zeros_like(x)
            ni, nj = int(nsol[i]), int(nsol[j])
            y[:ni, :nj] = sol[i, :ni] @ x @ sol[j, :nj].T
            basis[b] = y.T
    return {"orth": orth, "basis": basis}


def _long(case):
    """The segments of the wave, one by one on dense matrices, would take over twenty seconds."""
    pairs = case["nch"] * (case["nch"] + 1) // 2
    return case["occupancy"] * pairs * (case["mk"] + 1) * case["ns"] ** 2 > 8e7


def exact(case, seed):
    kind = case["kind"]
    if kind == "structures":
        return None  # the one-electron and bound structures have no plain form of this length
    if kind in ("assemble", "replay"):
        if _long(case):
            return None
        w = _workload(case, seed)
        pq = w.pq
        if kind == "replay":
            rng = np.random.Generator(np.random.Philox(seed + 77))
            pq = w.pq * (1.0 + rng.uniform(-1e-3, 1e-3, w.pq.shape))
        hch, acf = _exact_wave(w, pq)
        if case.get("out") in ("host", "host-window"):
            hch = hch.permute(2, 1, 0).cpu().numpy()  # (row, column, block)
            if case["out"] == "host-window":
                hch = hch.reshape(-1, order="F")
        return {"hch": hch, "acf": acf}
    if kind == "batch":
        if sum(_long(dict(case, ns=case["ns"] + i * case["ns_step"], nch=case["nch"] + i))
               for i in range(case["nwaves"])):
            return None
        got = []
        for i in range(case["nwaves"]):
            w = _workload(dict(case, ns=case["ns"] + i * case["ns_step"], nch=case["nch"] + i),
                          seed + i)
            got.append(_exact_wave(w, w.pq))
        return {"hch": [x for x, _ in got], "acf": [y for _, y in got]}
    if kind == "energy":
        e, g = _exact_energy(_energy(case, seed))
        return {"energy": e, "gradient": g}
    if kind == "scf":
        return _exact_scf(case, seed)
    return _exact_writeout(case, seed)
