"""The work that users of this framework have it do, as cases to time.

A case is one call (or one small sequence of calls) of the public Python API on
seeded synthetic data: founder-mosaic panels, targets that are mosaics of panel
haplotypes, typed at an array's sites or each at its own. Every pass goes
through ``swiftimpute_b200.engine``.

kind     what runs
impute   Engine.impute_device on device buffers (``mode``: the reference's
         first-gap transition, per-gap transitions, or target-aware selection)
host     Engine.impute on host arrays, copies inside the call
plan     an uneven batch (slices of the panel, mixed L) replayed as one graph
index    Engine.pbwt_build and the selection read from it

``out``  d: dosage, h: phased alleles, p: P(hap=1)
``spacing``  base pairs between markers (1e8 bp = 1 Morgan, the map rule)
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from swiftimpute_b200 import _native as native
from swiftimpute_b200 import synth_device
from swiftimpute_b200.engine import Engine

NE = 20_000


def _impute(name, N, M, B, L, every, spacing=500_000, out="dh", typed="array", sampling="argmax", mode="first_gap",
            kind="impute"):
    c = dict(kind=kind, N=N, M=M, B=B, L=L, every=every, spacing=spacing, out=out, typed=typed, sampling=sampling,
             mode=mode)
    return dict(name=name, **c) if name else c


def listed():
    return [
        # one target of the small amplicon panel: a single sample imputed as it arrives
        _impute("one_target", 4432, 1644, 1, 8, 5),
        # the reference's published run: its whole small cohort in one call
        _impute("plain_small", 4432, 1644, 444, 8, 5),
        # phased draws and haplotype probabilities of targets that are each typed at their own
        # sites, on a real-density map; no size a multiple of anything
        _impute("sampled_own_sites", 1009, 7919, 131, 5, 11, spacing=1000, out="dhp", typed="own", sampling="philox"),
        # the headline workload: a cohort on one array, every output the default call has
        _impute("dense_cohort", 4432, 50_000, 10_000, 8, 17),
        # a cohort on a sequencing-density map, rows of odd length
        _impute("dense_map", 4432, 30_011, 2003, 8, 16, spacing=1000),
        # a large panel with more states, as used for rare variants
        _impute("large_panel_16", 20_000, 20_000, 4000, 16, 20),
        # the most states, phased alleles alone (what the reference's VCF holds)
        _impute("states_32_gt", 6000, 6007, 1500, 32, 10, spacing=1000, out="h"),
        # per-gap transitions: a genetic map followed marker by marker
        _impute("per_gap", 4432, 20_000, 1000, 8, 16, spacing=1000, mode="per_gap"),
        # slots chosen per target from the panel
        _impute("target_slots", 1024, 4003, 512, 8, 10, spacing=1000, mode="target"),
        # host arrays in, host arrays out: a script without device buffers
        _impute("host_arrays", 4432, 20_000, 500, 8, 17, kind="host"),
        # many regions of different length and L in one graph launch: a service's fixed batch
        dict(name="uneven_plan", kind="plan", N=8000, M=24_000, regions=24, jobs=600, longest=8000, every=20,
             spacing=500_000),
        # a panel arrives: its index, and the slots of every marker
        dict(name="index", kind="index", N=4432, M=50_000, L=8),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choices(["typed", "per_gap", "target", "host", "plan", "index"], [10, 2, 1, 1, 2, 2])[0]
    if kind == "index":
        N = _log(rng, 300, 40_000)
        return dict(kind="index", N=N, M=_log(rng, 1000, min(50_000, 220_000_000 // N)), L=rng.randint(2, 32))
    spacing = rng.choice([500_000, 100_000, 1000, 1000])
    every = rng.randint(4, 40)
    if kind == "plan":
        longest = _log(rng, 600, 8000)
        return dict(kind="plan", N=_log(rng, 300, 10_000), M=3 * longest, regions=rng.randint(1, 30),
                    jobs=_log(rng, 8, 800), longest=longest, every=every, spacing=spacing)
    N = _log(rng, 200, 20_000)
    M = _log(rng, 500, min(50_000, 220_000_000 // N))
    L = rng.choice([4, 8, 8, 8, 16, 32, rng.randint(2, 31)])
    if kind == "typed":
        B = _log(rng, 1, min(10_000, 120_000_000 // M))
        return _impute(None, N, M, B, L, every, spacing, rng.choice(["dh", "dh", "h", "d", "dhp"]),
                       rng.choice(["array", "array", "array", "own"]), rng.choice(["argmax", "argmax", "philox"]))
    if kind == "per_gap":
        M = min(M, 20_000)
        return _impute(None, N, M, _log(rng, 1, min(3000, 20_000_000 // M)), L, every, spacing, "dh", mode="per_gap")
    if kind == "target":
        N, M = min(N, 3000), min(M, 6000)
        return _impute(None, N, M, _log(rng, 1, 1000), min(L, N), every, spacing, "dh", mode="target")
    return _impute(None, N, M, _log(rng, 1, max(2, 10_000_000 // M)), L, every, spacing, "dh", kind="host")


# ---------------------------------------------------------------- inputs


def _panel(case, seed):
    return synth_device.make_panel(case["M"], case["N"], 100, seed=seed)


def _positions(case):
    return 1 + np.arange(case["M"], dtype=np.uint64) * np.uint64(case["spacing"])


def _codes(case, panel, seed):
    """Genotype codes [B][M] on the device, 3 at untyped markers."""
    if case["typed"] == "array":
        return synth_device.make_targets(panel, case["B"], case["every"], seed=seed)
    codes = synth_device.make_targets(panel, case["B"], 1, seed=seed)  # every marker, then each target its own sites
    g = torch.Generator(device="cuda").manual_seed(seed + 7)
    keep = torch.rand(codes.shape, generator=g, device="cuda") < 1.0 / case["every"]
    return torch.where(keep, codes, torch.full_like(codes, 3))


def _batch(case, panel, seed):
    """Regions (begin, end, L, origin) and jobs (region, codes on the host, sample id) of an uneven batch."""
    rng = random.Random(case["jobs"])  # the batch's layout is the case's, its genotypes are the seed's
    M = case["M"]
    regions = []
    for _ in range(case["regions"]):
        n = _log(rng, 500, case["longest"])
        a = rng.randint(0, M - n)
        regions.append((a, a + n, rng.choice([4, 8, 16]), native.INDEX_REGION))
    pool = synth_device.make_targets(panel, 256, case["every"], seed=seed).cpu().numpy()
    jobs = []
    for j in range(case["jobs"]):
        r = rng.randrange(case["regions"])
        jobs.append((r, pool[rng.randrange(256), regions[r][0]:regions[r][1]], j))
    return regions, jobs


def _params(case):
    return native.default_params(
        num_states=case["L"], ne=NE,
        transition_mode=native.TRANS_PER_GAP if case["mode"] == "per_gap" else native.TRANS_MATRIX0,
        selection_kind=native.SEL_TARGET if case["mode"] == "target" else native.SEL_AUTO,
        sampling=native.SAMPLE_PHILOX if case["sampling"] == "philox" else native.SAMPLE_ARGMAX)


_stream = None


def _user_stream():
    """The stream the program puts its device work on, one call after the other."""
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    return _stream.cuda_stream


def prepare(case, seed):
    panel = _panel(case, seed)
    eng = Engine(0)
    eng.upload_panel(panel.cpu().numpy())
    st = {"case": case, "eng": eng}
    if case["kind"] == "index":
        return st
    eng.set_map(_positions(case))
    if case["kind"] == "plan":
        regions, jobs = _batch(case, panel, seed)
        st["plan"] = eng.plan(regions, jobs, native.default_params(ne=NE),
                              max_anchors=case["longest"] // case["every"] + 2)
        return st
    eng.pbwt_build(store_index=case["mode"] == "target")
    st["params"] = _params(case)
    codes = _codes(case, panel, seed)
    if case["kind"] == "host":
        st["codes"] = codes.cpu().numpy()
        return st
    B, M = case["B"], case["M"]
    st["codes"] = codes
    if "d" in case["out"]:
        st["dosage"] = torch.empty((B, M), dtype=torch.float32, device="cuda")
    if "p" in case["out"]:
        st["hap_prob"] = torch.empty((B, M, 2), dtype=torch.float32, device="cuda")
    if "h" in case["out"]:
        st["haps"] = torch.empty((B, 2, M), dtype=torch.uint8, device="cuda")
    return st


def run(st):
    case, eng = st["case"], st["eng"]
    if case["kind"] == "index":
        eng.pbwt_build()
        return {"slots": eng.select_states(case["L"])}
    if case["kind"] == "plan":
        plan = st["plan"]
        plan.launch(graph=True, stream=_user_stream())
        return {"dosage": plan.d_dos, "haps": plan.d_haps}
    if case["kind"] == "host":
        return eng.impute(st["codes"], st["params"])
    ptr = {k: st[k].data_ptr() if k in st else None for k in ("dosage", "hap_prob", "haps")}
    eng.impute_device(st["codes"].data_ptr(), case["B"], st["params"], ptr["dosage"], ptr["hap_prob"], ptr["haps"],
                      stream=_user_stream())
    return {k: st[k] for k in ptr if k in st}


def _shape(case):
    """(cells, slots per cell) of a pass; an uneven batch by its expected length."""
    if case["kind"] == "plan":
        lo, hi = math.log(500), math.log(case["longest"])
        mean = (case["longest"] - 500) / (hi - lo) if hi > lo else 500
        return case["jobs"] * mean, 28 / 3
    return case["B"] * case["M"], case["L"]


def work(case):
    if case["kind"] == "index":
        # the panel's bits in, the slots of every marker out
        return {"bytes": case["M"] * (case["N"] / 8 + case["L"] * 8), "flops": 0}
    cells, L = _shape(case)
    per = 1 + sum({"d": 4, "h": 2, "p": 8}[x] for x in case.get("out", "dh"))  # the code in, the outputs out
    # per slot and cell: alpha and beta (two operations each), their product, the sum and the weighing by alleles
    flops = cells * L * 8
    if case.get("mode") in ("per_gap", "target"):
        flops += cells * L * 6  # both recursions step every marker
    return {"bytes": cells * per, "flops": flops}


# ---------------------------------------------------------------- the same in 64 bits


def _orders(panel):
    """The PBWT order after each marker: zeros first, each side in the order before."""
    order = np.arange(panel.shape[1])
    for row in panel:
        bits = row[order] != 0
        order = np.concatenate([order[~bits], order[bits]])
        yield order


def _slots(panel, L):
    """Haplotypes of the L slots [M][L] at the reference selection's positions of each order."""
    M, N = panel.shape
    use = np.arange(L) % N
    if L <= 32 and N <= 10_000:
        n = min(4, (N + 31) // 32, L)
        at = 32 * np.arange(n)
    else:
        n = min(N, L)
        at = np.arange(n)
    out = np.tile(use, (M, 1))
    for m, order in enumerate(_orders(panel)):
        out[m, :n] = order[at]
    return out


def _target_slots(panel, codes, L):
    """Slots [M][B][L] that follow each target through the orders."""
    M, N = panel.shape
    B = codes.shape[0]
    p = np.zeros(B, np.int64)
    before = np.arange(N)
    out = np.empty((M, B, L), np.int64)
    for m, order in enumerate(_orders(panel)):
        bits = panel[m][before].astype(np.int64)
        zeros = np.concatenate([[0], np.cumsum(1 - bits)])
        g = codes[:, m]
        one = np.where(g == 0, 0, np.where(g == 2, 1, bits[np.minimum(p, N - 1)]))
        p = np.where(one == 1, zeros[N] + p - zeros[p], zeros[p])
        first = np.clip(p - L // 2, 0, N - L)
        out[m] = order[first[:, None] + np.arange(L)[None, :]]
        before = order
    return out


def _transitions(pos, per_gap):
    """(c, delta) into each marker: T = c 11' + delta I, from the float log10 weights."""
    d = np.diff(pos.astype(np.float64) / 1e8)
    r = 1.0 - np.exp(-4.0 * NE * d * 4.0)
    stay = np.exp(np.float32(np.log10((1.0 - r) + r / (2 * NE))).astype(np.float64))
    off = np.exp(np.float32(np.log10(r / (2 * NE))).astype(np.float64))
    if not per_gap:
        off, stay = np.full_like(off, off[0]), np.full_like(stay, stay[0])
    return np.concatenate([[1.0], off]), np.concatenate([[0.0], stay - off])


def _posterior(panel, pos, codes, slots, per_gap=False):
    """Expected alleles [M][B][2] (of both haplotypes) under softmax(alpha + beta), FP64 on the device.

    slots [M][L], or [M][B][L] per target. Every logsumexp chain of beta starts
    at -999, so beta carries a floor of e^-999; a call that no slot matches
    scales every slot by e^-999.
    """
    M, N = panel.shape
    B = codes.shape[0]
    dev = codes.device
    P = torch.from_numpy(panel).to(dev)
    S = torch.from_numpy(slots).to(dev)
    shared = S.dim() == 2
    a0 = torch.gather(P, 1, S.reshape(M, -1)).reshape(S.shape).to(torch.float64)
    a1 = torch.gather(P, 1, ((S + 1) % N).reshape(M, -1)).reshape(S.shape).to(torch.float64)
    L = S.shape[-1]
    c, delta = _transitions(pos, per_gap)
    codes_t = codes.t().contiguous()
    typed = (codes_t < 3).any(1).cpu().numpy()

    def emission(m):
        g = codes_t[m][:, None]
        match = (a0[m] + a1[m]) == g
        hit = match.any(1, keepdim=True)
        none = (~hit) & (g < 3)
        return torch.where(hit, match, torch.ones_like(match)).to(torch.float64), none.to(torch.float64)

    E = {m: emission(m) for m in np.nonzero(typed)[0]}
    alpha = torch.empty((M, B, L), dtype=torch.float64, device=dev)
    for m in range(M):
        a = alpha[m]
        if m == 0:
            a.fill_(1.0)
        else:
            torch.mul(alpha[m - 1], delta[m], out=a)
            a.add_(alpha[m - 1].sum(1, keepdim=True), alpha=c[m])
        if typed[m]:
            a.mul_(E[m][0])
        if m % 16 == 0 or m + 1 == M:
            a.div_(a.sum(1, keepdim=True))
    out = torch.empty((M, B, 3), dtype=torch.float64, device=dev)
    if shared:
        weigh = torch.stack([torch.ones_like(a0), a0, a1], -1)  # [M][L][3]
    beta = torch.ones((B, L), dtype=torch.float64, device=dev)
    unit = torch.zeros((B, 1), dtype=torch.float64, device=dev)  # log of beta's unit
    for m in range(M - 1, -1, -1):
        if m + 1 < M:
            if typed[m + 1]:
                e, none = E[m + 1]
                beta = beta * e
                unit = unit - 999.0 * none
            beta = torch.add(beta * delta[m + 1], beta.sum(1, keepdim=True), alpha=c[m + 1])
            top = unit.clamp(min=-999.0)
            beta = beta * torch.exp(unit - top) + torch.exp(-999.0 - top)
            unit = top
            if m % 4 == 0:
                s = beta.sum(1, keepdim=True)
                beta = beta / s
                unit = unit + torch.log(s)
        p = alpha[m] * beta
        if shared:
            torch.matmul(p, weigh[m], out=out[m])
        else:
            out[m, :, 0] = p.sum(1)
            out[m, :, 1] = (p * a0[m]).sum(1)
            out[m, :, 2] = (p * a1[m]).sum(1)
    return out[..., 1:] / out[..., :1]


def exact(case, seed):
    if case["kind"] == "index":
        return None  # whole numbers only
    if case.get("out", "dh") == "h" or (case["kind"] != "plan" and case["B"] * case["M"] * case["L"] > 5e9):
        return None
    dev_panel = _panel(case, seed)
    panel = dev_panel.cpu().numpy()
    pos = _positions(case)
    if case["kind"] == "plan":
        regions, jobs = _batch(case, dev_panel, seed)
        flat = [None] * len(jobs)
        for r, (a, b, L, _) in enumerate(regions):
            mine = [j for j, job in enumerate(jobs) if job[0] == r]
            if not mine:
                continue
            codes = torch.from_numpy(np.stack([jobs[j][1] for j in mine])).cuda()
            q = _posterior(panel[a:b], pos[a:b], codes, _slots(panel[a:b], L))
            for j, x in zip(mine, q.sum(-1).t()):
                flat[j] = x
        return {"dosage": torch.cat(flat), "haps": None}
    codes = _codes(case, dev_panel, seed)
    slots = _target_slots(panel, codes.cpu().numpy(), case["L"]) if case["mode"] == "target" else _slots(panel, case["L"])
    q = _posterior(panel, pos, codes, slots, case["mode"] == "per_gap").transpose(0, 1).contiguous()
    out = {"haps": None}
    if "d" in case["out"]:
        out["dosage"] = q.sum(-1)
    if "p" in case["out"]:
        out["hap_prob"] = q
    return out
