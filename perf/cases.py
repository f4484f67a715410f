"""The work that a user of libcc_b200 has it do, as cases that can be timed.

Every case is one pass through the public entry points: the (T) plan in its
native FP64 and emulated forms, a whole call on host arrays, a new system on a
kept plan, the gradient, a batch of uneven systems and the two CCSD
T1-dressing routines.  ``exact`` evaluates the same quantities in float64 from
their definitions with plain torch.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from libcc_b200 import _native, api, batch, shard

MEM_DEVICE = 1
INPUTS = ("eh", "ep", "t1", "t2", "vm", "voe", "vvvo")


# ---------------------------------------------------------------------------- cases

def listed():
    return [
        # water in aug-cc-pVDZ: the smallest published system; sixteen tuples, launch latency counts
        {"name": "fp64-no4-nu36", "kind": "forward", "form": "fp64", "vvvo": "auto", "no": 4, "nu": 36,
         "dist": "normal", "rank": 0, "world": 1},
        # a mid-size molecule on one GPU in the native form
        {"name": "fp64-no12-nu120", "kind": "forward", "form": "fp64", "vvvo": "auto", "no": 12, "nu": 120,
         "dist": "normal", "rank": 0, "world": 1},
        # one rank's share of a large system (i>j>k and degenerate tuples) in the native form
        {"name": "fp64-no24-nu320-r14of16", "kind": "forward", "form": "fp64", "vvvo": "auto", "no": 24, "nu": 320,
         "dist": "log", "rank": 14, "world": 16},
        # an odd-sized small molecule, emulated, digits calibrated to the default energy target
        {"name": "int8-no9-nu83", "kind": "forward", "form": "int8", "vvvo": "auto", "no": 9, "nu": 83,
         "dist": "normal", "rank": 0, "world": 1},
        # one rank's share of a large system, emulated to a relative energy target
        {"name": "int8rel-no24-nu320-r6of8", "kind": "forward", "form": "int8@2.1e-7", "vvvo": "auto", "no": 24,
         "nu": 320, "dist": "log", "rank": 6, "world": 8},
        # a new geometry on a kept emulated plan: inputs from the device, digit calibration, all tuples
        {"name": "int8-new-no16-nu200", "kind": "fresh", "form": "int8", "vvvo": "auto", "no": 16, "nu": 200,
         "dist": "normal", "rank": 0, "world": 1},
        # the whole driver on host arrays, as a Fortran program calls it: plan, upload, (T), release
        {"name": "call-no8-nu72", "kind": "call", "no": 8, "nu": 72, "dist": "normal"},
        # energy and its gradient with respect to every input
        {"name": "grad-no12-nu120", "kind": "grad", "keep_w": False, "no": 12, "nu": 120, "dist": "normal"},
        # many small molecules together, native form
        {"name": "batch-fp64-24", "kind": "batch", "form": "fp64", "systems": 24, "no_lo": 3, "no_hi": 12,
         "nu_lo": 24, "nu_hi": 140, "shapes": 100},
        # the same, emulated with a digit count per system
        {"name": "batch-int8-24", "kind": "batch", "form": "int8", "systems": 24, "no_lo": 3, "no_hi": 12,
         "nu_lo": 24, "nu_hi": 140, "shapes": 100},
        # CCSD T1-dressing terms inside an iteration, everything on the device
        {"name": "ccsd2931-no24-nu320", "kind": "ccsd2931", "no": 24, "nu": 320},
        {"name": "ccsd3235-no16-nu200", "kind": "ccsd3235", "no": 16, "nu": 200},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["forward", "forward", "forward", "fresh", "call", "grad", "batch", "ccsd2931", "ccsd3235"])
    if kind == "batch":
        return {"kind": kind, "form": rng.choice(["fp64", "int8"]), "systems": _log_int(rng, 4, 24), "no_lo": 3,
                "no_hi": rng.randint(6, 12), "nu_lo": 24, "nu_hi": rng.randint(60, 140),
                "shapes": rng.randint(0, 10 ** 6)}
    if kind in ("ccsd2931", "ccsd3235"):
        return {"kind": kind, "no": _log_int(rng, 3, 24), "nu": _log_int(rng, 24, 320 if kind == "ccsd2931" else 240)}
    if kind == "call":
        return {"kind": kind, "no": _log_int(rng, 3, 12), "nu": _log_int(rng, 24, 120), "dist": "normal"}
    if kind == "grad":
        return {"kind": kind, "keep_w": rng.random() < 0.3, "no": _log_int(rng, 3, 12), "nu": _log_int(rng, 20, 120),
                "dist": "normal"}
    form = rng.choice(["fp64", "int8", "int8@2.1e-7", "int8:4"]) if kind == "forward" else \
        rng.choice(["fp64", "int8", "int8@2.1e-7"])
    case = {"kind": kind, "form": form, "vvvo": "auto", "no": _log_int(rng, 3, 24), "nu": _log_int(rng, 20, 320),
            "dist": rng.choice(["normal", "log"]), "rank": 0, "world": 1}
    if form == "fp64" and rng.random() < 0.25:
        case["vvvo"] = "packed"
    # a large system is shared out over ranks, as it would be
    limit = 1.0e13 if form == "fp64" else 2.5e13
    while _tuple_flops(case["no"], case["nu"]) * sum(shard.tuple_costs(case["no"])) / case["world"] > limit:
        case["world"] *= 2
    case["rank"] = rng.randrange(case["world"])
    return case


# ---------------------------------------------------------------------------- inputs

def _values(gen, shape, dist):
    if dist == "normal":
        return torch.empty(shape, dtype=torch.float64, device="cuda").normal_(0.0, 0.05, generator=gen)
    x = torch.empty(shape, dtype=torch.float64, device="cuda").uniform_(-6.0, 0.0, generator=gen)
    torch.pow(10.0, x, out=x)
    sign = torch.empty(shape, dtype=torch.float32, device="cuda").uniform_(-1.0, 1.0, generator=gen)
    return x.mul_(torch.where(sign < 0, -1.0, 1.0))


def _mirror(x):
    """x[j][i][b][a] made symmetric under (a,i) <-> (b,j), keeping one half's values."""
    no, nu = x.shape[0], x.shape[2]
    o, v = torch.arange(no, device="cuda"), torch.arange(nu, device="cuda")
    key = v[:, None] * no + o[None, :]  # [virtual][occupied]
    ai = key.t()[None, :, None, :]      # [.][i][.][a]
    bj = key.t()[:, None, :, None]      # [j][.][b][.]
    return torch.where(ai <= bj, x, x.permute(1, 0, 3, 2))


def _system(no, nu, dist, seed):
    """(T) inputs in the reference's Fortran layouts, as flat device tensors."""
    gen = torch.Generator(device="cuda").manual_seed(seed)

    def uniform(n, lo, hi):
        return torch.empty(n, dtype=torch.float64, device="cuda").uniform_(lo, hi, generator=gen).sort().values

    eh, ep = uniform(no, -1.4, -0.4), uniform(nu, 0.1, 4.0)
    t1 = torch.empty(nu * no, dtype=torch.float64, device="cuda").normal_(0.0, 0.005, generator=gen)
    t2 = _mirror(_values(gen, (no, no, nu, nu), dist))  # [j][i][b][a]
    t2 /= (ep[None, None, None, :] + ep[None, None, :, None] - eh[None, :, None, None] - eh[:, None, None, None])
    voe = _mirror(_values(gen, (no, no, nu, nu), dist))
    v = _values(gen, (no, no, nu, no), dist)            # VM [y][x][c][l] = (c x|l y), symmetric in l, y
    o = torch.arange(no, device="cuda")
    vm = torch.where((o[:, None] <= o[None, :])[:, None, None, :], v, v.permute(3, 1, 2, 0))
    vvvo = _values(gen, (nu * no, nu * (nu + 1) // 2), dist)
    return {"eh": eh, "ep": ep, "t1": t1, "t2": t2.contiguous().view(-1), "vm": vm.contiguous().view(-1),
            "voe": voe.contiguous().view(-1), "vvvo": vvvo.view(-1)}


def _shapes(case):
    rng = np.random.default_rng(case["shapes"])
    return [(int(rng.integers(case["no_lo"], case["no_hi"] + 1)), int(rng.integers(case["nu_lo"], case["nu_hi"] + 1)))
            for _ in range(case["systems"])]


def _ccsd_inputs(case, seed):
    no, nu = case["no"], case["nu"]
    gen = torch.Generator(device="cuda").manual_seed(seed)

    def normal(n, sigma):
        return torch.empty(n, dtype=torch.float64, device="cuda").normal_(0.0, sigma, generator=gen)

    n4 = no * nu * nu * no
    d = {"o1": normal(no * nu, 0.05), "t2": normal(n4, 0.05), "vvvo": normal(nu * (nu + 1) // 2 * nu * no, 0.05)}
    if case["kind"] == "ccsd2931":
        d.update(vl=normal(n4, 0.05), vr=normal(n4, 0.05))
    else:
        d.update(o2=normal(n4, 0.05), vm=normal(no ** 3 * nu, 0.05))
    return d


# ---------------------------------------------------------------------------- prepare and run

def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def prepare(case, seed):
    kind = case["kind"]
    state = {"case": case}
    if kind in ("forward", "fresh"):
        state["range"] = shard.shard_of(case["no"], case["rank"], case["world"])
        state["plan"] = api.TriplesPlan.for_form(case["no"], case["nu"], case["form"], vvvo=case["vvvo"])
        sys = _system(case["no"], case["nu"], case["dist"], seed)
        if kind == "forward":
            state["plan"].set_inputs(**sys)
        else:
            state["inputs"] = sys
    elif kind == "call":
        sys = _system(case["no"], case["nu"], case["dist"], seed)
        state["inputs"] = {k: v.cpu().numpy() for k, v in sys.items()}
    elif kind == "grad":
        state["plan"] = api.TriplesPlan(case["no"], case["nu"], keep_w=case["keep_w"])
        sys = _system(case["no"], case["nu"], case["dist"], seed)
        state["plan"].set_inputs(**sys)
        state["grads"] = {k: torch.empty_like(v) for k, v in sys.items()}
    elif kind == "batch":
        shapes = _shapes(case)
        b = batch.TriplesBatch(shapes, form=case["form"])
        for s, (no, nu) in enumerate(shapes):
            sys = _system(no, nu, "normal", seed * 1000 + s)
            torch.cuda.synchronize()
            _native.check(_native.load().ccT_batch_set_inputs(b._h, s, *[_ptr(sys[k]) for k in INPUTS], MEM_DEVICE),
                          "ccT_batch_set_inputs")
        state["batch"] = b
    else:
        state["inputs"] = _ccsd_inputs(case, seed)
        state["work"] = {k: torch.empty_like(state["inputs"][k]) for k in ("t2", "o2", "vm") if k in state["inputs"]}
        if kind == "ccsd3235":
            state["work"]["rl"] = torch.empty_like(state["inputs"]["t2"])
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "forward":
        return state["plan"].forward(*state["range"])
    if kind == "fresh":
        state["plan"].set_inputs(**state["inputs"])
        return state["plan"].forward(*state["range"])
    if kind == "call":
        return api.cc_triples(case["no"], case["nu"], *[state["inputs"][k] for k in INPUTS])
    if kind == "grad":
        plan, g = state["plan"], state["grads"]
        energies = plan.forward()
        _native.check(_native.load().ccT_backward(plan._h, 0, plan.num_tuples, *[_ptr(g[k]) for k in INPUTS],
                                                  MEM_DEVICE), "ccT_backward")
        return energies, g
    if kind == "batch":
        b = state["batch"]
        ets, etd = b.forward()
        return ets, etd, [b.v1(s) for s in range(len(b))]
    # the CCSD routines update their arrays in place; the iteration's own copies go in
    lib, x, w = _native.load(), state["inputs"], state["work"]
    for k in w:
        if k in x:
            w[k].copy_(x[k])
    if kind == "ccsd2931":
        _native.check(lib.ccT_ccsd_terms_29_31(case["no"], case["nu"], _ptr(x["o1"]), _ptr(w["t2"]), _ptr(x["vl"]),
                                               _ptr(x["vr"]), _ptr(x["vvvo"]), MEM_DEVICE), "ccT_ccsd_terms_29_31")
        return w["t2"]
    _native.check(lib.ccT_ccsd_terms_32_35(case["no"], case["nu"], _ptr(x["o1"]), _ptr(w["o2"]), _ptr(w["t2"]),
                                           _ptr(w["vm"]), _ptr(w["rl"]), _ptr(x["vvvo"]), MEM_DEVICE),
                  "ccT_ccsd_terms_32_35")
    return w["t2"], w["o2"], w["vm"], w["rl"]


# ---------------------------------------------------------------------------- work

def _tuple_flops(no, nu):
    return 12.0 * nu ** 3 * (no + nu)


def _system_elements(no, nu):
    return no + nu + no * nu + 2 * nu * nu * no * no + no ** 3 * nu + nu * (nu + 1) // 2 * nu * no


def work(case):
    kind = case["kind"]
    if kind == "batch":
        shapes = _shapes(case)
        return {"bytes": 8.0 * sum(_system_elements(o, v) + o * v for o, v in shapes),
                "flops": sum(_tuple_flops(o, v) * sum(shard.tuple_costs(o)) for o, v in shapes)}
    no, nu = case["no"], case["nu"]
    n4, nutr = no * nu * nu * no, nu * (nu + 1) // 2
    if kind == "ccsd2931":  # the O1 contractions with VVVO, VL and VR, then the two O1 products per T2 element
        return {"bytes": 8.0 * (4 * n4 + no * nu + nutr * nu * no),
                "flops": 2.0 * no * no * nu ** 3 + 8.0 * no ** 3 * nu * nu}
    if kind == "ccsd3235":
        return {"bytes": 8.0 * (5 * n4 + no * nu + 2 * no ** 3 * nu + nutr * nu * no),
                "flops": 2.0 * no * no * nu ** 3 + 2.0 * no ** 3 * nu ** 3}
    if kind in ("call", "grad"):
        flops = _tuple_flops(no, nu) * sum(shard.tuple_costs(no))
        n = _system_elements(no, nu)
        # the gradient: the W build again and the products with both of its operands
        return {"bytes": 8.0 * (n + no * nu + (n if kind == "grad" else 0)),
                "flops": flops * (3.0 if kind == "grad" else 1.0)}
    begin, end = shard.shard_of(no, case["rank"], case["world"])
    tuples = _tuples(no)[begin:end]
    flops = _tuple_flops(no, nu) * sum(0.5 if i == j or j == k else 1.0 for i, j, k in tuples)
    # the slices of the range: VVVO and T2 of every index met, VM and VOE of every pair
    occ = {x for t in tuples for x in t}
    pairs = {(x, y) for t in tuples for a, x in enumerate(t) for b, y in enumerate(t) if a != b}
    n = len(occ) * nutr * nu + len(pairs) * (2 * nu * nu + no * nu) + no + nu + 2 * no * nu
    if kind == "fresh":
        n = max(n, _system_elements(no, nu) + no * nu)
    return {"bytes": 8.0 * n, "flops": flops}


# ---------------------------------------------------------------------------- exact values

def _tuples(no):
    """The plan's tuple order: i>j>k, then per i and j<i the (i,j,j) and (i,i,j) tuples."""
    out = [(i, j, k) for i in range(no) for j in range(i) for k in range(j)]
    for i in range(no):
        for j in range(i):
            out += [(i, j, j), (i, i, j)]
    return out


class _Views:
    """The inputs by index: T2(a,b,i,j) = t2[i][j][a,b], VM(l,c,x,y) = vm[x][y][l,c], VOE(a,b,i,j) =
    voe[i][j][a,b], (d q|p x) = v[x][p,q,d], T1(i,a) = t1[i,a]."""

    def __init__(self, no, nu, s, occupied, grad=False):
        def leaf(t):
            return t.contiguous().requires_grad_(grad)

        self.no, self.nu = no, nu
        self.eh, self.ep = leaf(s["eh"].clone()), leaf(s["ep"].clone())
        self.t1 = leaf(s["t1"].view(nu, no).t().clone())
        t2, voe, vm = s["t2"].view(no, no, nu, nu), s["voe"].view(no, no, nu, nu), s["vm"].view(no, no, nu, no)
        r = range(no)
        self.t2 = [[leaf(t2[j, i].t()) for j in r] for i in r]
        self.voe = [[leaf(voe[j, i].t()) for j in r] for i in r]
        self.vm = [[leaf(vm[y, x].t()) for y in r] for x in r]
        a = torch.arange(nu, device="cuda")
        hi, lo = torch.maximum(a[:, None], a[None, :]), torch.minimum(a[:, None], a[None, :])
        tri = (hi * (hi + 1) // 2 + lo).view(-1)
        packed = s["vvvo"].view(no, nu, -1)
        self.v = {x: leaf(packed[x][:, tri].view(nu, nu, nu)) for x in occupied}


def _tuple_energy(s, i, j, k, weight):
    """Weighted E[4] of one tuple and its v1 columns for i, j and k."""
    nu = s.nu

    def h(x, y, z):  # sum_d (d q|p x) T2(s,d,y,z) - sum_l T2(p,q,l,x) VM(l,s,z,y), as [p,q,s]
        r = (s.v[x].reshape(nu * nu, nu) @ s.t2[y][z].t()).view(nu, nu, nu)
        t = torch.stack([s.t2[l][x] for l in range(s.no)], dim=-1)
        return r - (t.view(nu * nu, s.no) @ s.vm[z][y]).view(nu, nu, nu)

    w = h(i, j, k)
    w = w + h(j, i, k).permute(1, 0, 2)
    w = w + h(i, k, j).permute(0, 2, 1)
    w = w + h(k, i, j).permute(1, 2, 0)
    w = w + h(j, k, i).permute(2, 0, 1)
    w = w + h(k, j, i).permute(2, 1, 0)
    a = torch.arange(nu, device="cuda")
    mask = torch.zeros(nu, nu, nu, dtype=torch.bool, device="cuda")
    mask[a, a, a] = True
    w = w.masked_fill(mask, 0.0)
    e = s.ep
    d = weight / (s.eh[i] + s.eh[j] + s.eh[k] - (e[:, None, None] + e[None, :, None] + e[None, None, :]))
    acb, bac, cba = w.permute(0, 2, 1), w.permute(1, 0, 2), w.permute(2, 1, 0)
    bca, cab = w.permute(2, 0, 1), w.permute(1, 2, 0)  # [a,b,c] -> w[b,c,a], w[c,a,b]
    e4 = ((8 * w - 4 * (acb + cba + bac) + 2 * (bca + cab)) * w * d).sum()

    def column(z, y, x):
        return (z * d).reshape(nu, nu * nu) @ s.voe[y][x].reshape(-1)

    vi = column((w - bac) * 2 - acb + bca, j, k) + column((acb - bca) * 2 - w + bac, k, j)
    vj = column((bac - w) * 2 - cab + cba, i, k) + column((cab - cba) * 2 - bac + w, k, i)
    vk = column((bca - acb) * 2 - cba + cab, i, j) + column((cba - cab) * 2 - bca + acb, j, i)
    return e4, vi, vj, vk


def _energies(no, nu, sys, tuples, grad=False):
    occ = sorted({x for t in tuples for x in t})
    with torch.set_grad_enabled(grad):
        s = _Views(no, nu, sys, occ, grad)
        v1 = torch.zeros(no, nu, dtype=torch.float64, device="cuda")
        etd = 0.0
        for i, j, k in tuples:
            e4, *cols = _tuple_energy(s, i, j, k, 0.5 if i == j or j == k else 1.0)
            if grad:
                (e4 + 2.0 * sum((s.t1[x] * c).sum() for x, c in zip((i, j, k), cols))).backward()
            etd += float(e4.detach())
            for x, c in zip((i, j, k), cols):
                v1[x] += c.detach()
    ets = 2.0 * float((s.t1.detach() * v1).sum())
    return s, (ets, etd, v1.view(-1).cpu().numpy())


def _gradients(s):
    no, nu = s.no, s.nu
    r = range(no)

    def g(t):
        return torch.zeros_like(t) if t.grad is None else t.grad

    a = torch.arange(nu, device="cuda")
    lower = a[:, None] >= a[None, :]
    vvvo = []
    for x in r:
        gv = g(s.v[x])  # [p,q,d], the packed entry is (q,d) and (d,q)
        full = gv + gv.transpose(1, 2)
        full[:, a, a] = gv[:, a, a]
        vvvo.append(full[:, lower])
    return {"eh": g(s.eh), "ep": g(s.ep), "t1": g(s.t1).t().reshape(-1),
            "t2": torch.stack([torch.stack([g(s.t2[i][j]).t() for i in r]) for j in r]).reshape(-1),
            "vm": torch.stack([torch.stack([g(s.vm[x][y]).t() for x in r]) for y in r]).reshape(-1),
            "voe": torch.stack([torch.stack([g(s.voe[i][j]).t() for i in r]) for j in r]).reshape(-1),
            "vvvo": torch.cat(vvvo).reshape(-1)}


def _full_vvvo(vvvo, no, nu, j):
    """(x y|z j) as [z,x,y]."""
    a = torch.arange(nu, device="cuda")
    hi, lo = torch.maximum(a[:, None], a[None, :]), torch.minimum(a[:, None], a[None, :])
    return vvvo.view(no, nu, -1)[j][:, (hi * (hi + 1) // 2 + lo).view(-1)].view(nu, nu, nu)


def _exact_2931(no, nu, d):
    o1 = d["o1"].view(nu, no)                                                   # [x][i]
    vl, vr = d["vl"].view(no, nu, nu, no), d["vr"].view(no, nu, no, nu)         # [j][y][x][k], [j][x][k][z]
    out = d["t2"].view(no, nu, nu, no).clone()                                  # [j][z][y][i]
    for j in range(no):
        x = torch.einsum("yzx,xi->zyi", _full_vvvo(d["vvvo"], no, nu, j), o1)   # (z x|y j) o1(i,x)
        p = torch.einsum("yxk,xi->yki", vl[j], o1)
        q = torch.einsum("xkz,xi->zki", vr[j], o1)
        x -= torch.einsum("zk,yki->zyi", o1, p) + torch.einsum("yk,zki->zyi", o1, q)
        out[j] += x
    return out.reshape(-1)


def _exact_3235(no, nu, d):
    o1 = d["o1"].view(nu, no)
    nou = no * nu
    t2 = d["t2"].view(nou, nou).t().contiguous().view(-1)
    o2 = d["o2"].view(no, nu, nu, no)                                           # O2(k,x,y,l) [l][y][x][k]
    o2b = o2.permute(0, 3, 1, 2).contiguous()                                   # [l][k][y][x]
    rows = o2b.view(no * no, nu * nu)
    vm = d["vm"].view(nu, no, no, no).transpose(2, 3).contiguous()              # [a][z][y][x] <- (y,x,z,a)
    rl = torch.empty(nu, no, no, nu, dtype=torch.float64, device="cuda")        # [y][i][j][z]
    for j in range(no):
        v = _full_vvvo(d["vvvo"], no, nu, j)                                    # (a y|x j) [x][a][y]
        rl[:, :, j, :] = torch.einsum("zxy,xi->yiz", v, o1)                     # (x y|z j) o1(i,x)
        b = v.permute(1, 2, 0).reshape(nu, nu * nu)                             # [a][y,x]
        vm[:, :, j, :] += (b @ rows.t()).view(nu, no, no)                       # vm(k,j,l,a) += T((k,l),(a,j))
    return t2, o2b.view(-1), vm.view(-1), rl.view(-1)


def exact(case, seed):
    kind = case["kind"]
    if kind == "ccsd2931":
        return _exact_2931(case["no"], case["nu"], _ccsd_inputs(case, seed))
    if kind == "ccsd3235":
        return _exact_3235(case["no"], case["nu"], _ccsd_inputs(case, seed))
    if kind == "batch":
        res = [_energies(no, nu, _system(no, nu, "normal", seed * 1000 + s), _tuples(no))[1]
               for s, (no, nu) in enumerate(_shapes(case))]
        return np.array([r[0] for r in res]), np.array([r[1] for r in res]), [r[2] for r in res]
    no, nu = case["no"], case["nu"]
    sys = _system(no, nu, case["dist"], seed)
    if kind == "grad":
        s, energies = _energies(no, nu, sys, _tuples(no), grad=True)
        return energies, _gradients(s)
    begin, end = shard.shard_of(no, case["rank"], case["world"]) if "world" in case else (0, len(_tuples(no)))
    return _energies(no, nu, sys, _tuples(no)[begin:end])[1]
