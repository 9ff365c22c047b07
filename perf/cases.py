"""Performance cases of the framework: what a user's program has it do, over the range of sizes.

Physics cases advance river networks generated by the configuration laws of `cmf_b200.synth`:
  plain  config 0: rivers and floodplains only (one 100x100 tile is 10,000 cells);
  full   config 1: bifurcation channels, levees on 10 % of cells, dams, 300k cells at scale 1;
  flood  config 1 with low banks under heavy runoff: about half of the cells are out of bank.
Every network starts near the balance of its mean runoff (Manning's normal depth in each channel,
flows reconstructed by the storage-only restart) and is run for a day before it is handed over, as
a program that resumes a simulation has it.  Emulator cases use the framework's 64-128-128-128-64
network with seeded weights.

A case is a dict of plain values: "kind" and the sizes that `prepare` reads.
"""
from __future__ import annotations

import functools
import os
import sys
import tempfile

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cama-flood_v4_b200"))

from cmf_b200 import HostModel, PhysicsBatch, PhysicsGPU, synth  # noqa: E402
from cmf_b200 import emulator as E  # noqa: E402

SPINUP = 24          # hours a network is run before a case begins
FIELDS = 4           # distinct hourly runoff fields a case goes round
STEP_FIELDS = ("outflw_aavg", "rivdph", "storge")
FULL_FIELDS = ("rivout_aavg", "fldout_aavg", "outflw_aavg", "rivvel_aavg", "storge_amax", "rivdph_amax",
               "rivdph", "flddph", "fldfrc", "fldare", "sfcelv", "storge")
MEAN_NT = 30         # adaptive sub-steps per hour (10 in the flooded basins to 47 on the global network)
CELL_BYTES = 316     # one cell's sub-step: state and maps read once, state written once


def _device():
    return torch.device("cuda", torch.cuda.current_device())


# ------------------------------------------------------------------------------------- the cases
def listed() -> list:
    return [
        # the smallest call: a regional river network coupled hour by hour with host arrays
        {"name": "step_10k_plain", "kind": "step", "law": "plain", "cells": 10_000, "members": 1},
        # a flood forecast: a few members of a basin in flood, every state field read back each hour
        {"name": "step_75k_flood_x4", "kind": "step", "law": "flood", "cells": 75_000, "members": 4, "fields": "full"},
        # the largest regional domain, one member
        {"name": "step_2m", "kind": "step", "law": "full", "cells": 2_000_000, "members": 1},
        # the global quarter-degree model, pipelined with its host: uploads and read-backs overlap the steps
        {"name": "pipeline_300k", "kind": "pipeline", "law": "full", "cells": 300_000, "members": 1, "hours": 6},
        # a runoff ensemble of it, forcing and results on the device
        {"name": "ensemble_300k_x16", "kind": "ensemble", "law": "full", "cells": 300_000, "members": 16},
        # regional domains of uneven size, each with its members, one launch per hour
        {"name": "batch_4_domains_x8", "kind": "batch", "law": "full", "cells": 180_000, "domains": 4, "members": 8},
        # six hours of gridded forcing through the input matrix, then the output averages of the interval
        {"name": "output_6h_27k_x2", "kind": "output", "law": "full", "cells": 27_000, "members": 2, "hours": 6},
        # one hour of an ensemble under the emulator
        {"name": "emu_hour_300k_x32", "kind": "emu_hour", "law": "full", "cells": 300_000, "members": 32},
        # the emulator's network alone: a small domain, and an ensemble
        {"name": "infer_27k_rows", "kind": "infer", "rows": 26_595},
        {"name": "infer_4m_rows", "kind": "infer", "rows": 4_194_304},
        # one training step: the usual batch, and a large one whose last rows are padding
        {"name": "train_16k", "kind": "train", "rows": 16_384, "valid": 16_384},
        {"name": "train_128k", "kind": "train", "rows": 131_072, "valid": 130_001},
    ]


def _spread(rng, lo: int, hi: int) -> int:
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng) -> dict:
    kind = rng.choice(["step", "step", "step", "ensemble", "pipeline", "batch", "output", "emu_hour", "infer", "train"])
    if kind == "infer":
        return {"kind": kind, "rows": _spread(rng, 1_000, 4_194_304)}
    if kind == "train":
        rows = 64 * _spread(rng, 16, 2048)
        return {"kind": kind, "rows": rows, "valid": rows - rng.randrange(64)}
    if kind == "batch":
        return {"kind": kind, "law": "full", "cells": _spread(rng, 20_000, 200_000), "domains": rng.randint(2, 5),
                "members": rng.randint(1, 8)}
    cells = _spread(rng, 5_000, 600_000)
    law = rng.choice(["plain", "full", "full", "flood"]) if kind == "step" else "full"
    most = {"step": 600_000, "pipeline": 600_000, "output": 100_000, "ensemble": 4_800_000, "emu_hour": 9_600_000}[kind]
    cells = min(cells, most)
    members = _spread(rng, 1, max(1, min(48, most // cells)))
    case = {"kind": kind, "law": law, "cells": cells, "members": members}
    if kind in ("pipeline", "output"):
        case["hours"] = rng.randint(3, 6)
    if kind == "step" and rng.random() < 0.3:
        case["fields"] = "full"
    return case


# ---------------------------------------------------------------------------------- the networks
def _spec(law: str, cells: int):
    if law == "plain":
        ny = max(8, int(round(cells ** 0.5)))
        nx = max(8, int(round(cells / ny)))
        return synth.CaseSpec(name="plain", nx=nx, ny=ny, land_frac=1.0, n_mouths=max(2, cells // 500), seed=cells % 1009,
                              dt=3600.0, ifrq_inp=24)
    spec = synth.spec_config1(seed=1 + cells % 1009, scale=(cells / 300_000.0) ** 0.5)
    if law == "flood":
        spec.rivhgt_scale = 0.15
        spec.fldhgt_inc_max = 0.6
    return spec


@functools.lru_cache(maxsize=8)
def _network(law: str, cells: int):
    """(host model, river storage of the normal depth at the mean runoff, mean runoff in mm/day)."""
    case = synth.make_case(_spec(law, cells))
    with tempfile.TemporaryDirectory() as d:
        synth.write_case(case, d)
        host = HostModel(d)
    mean = 2.0 if law != "flood" else 5.0
    q = np.maximum(host.grid_to_seq(case.uparea), 1.0) * mean * 1e3 / 86400.0          # m3/s
    nxt = host.map("i1next") - 1
    elv, dst = host.map("elevtn"), host.map("nxtdst")
    slope = np.full(q.size, 1e-4)
    river = nxt >= 0
    slope[river] = np.clip((elv[river] - elv[nxt[river]]) / dst[river], 1e-5, 1e-2)
    wth = host.map("rivwth")
    depth = (q * host.map("rivman") / (wth * np.sqrt(slope))) ** 0.6
    return host, np.maximum(host.initial_state()["rivsto"], wth * host.map("rivlen") * depth), mean


def _runoff(host, mean: float, members: int, seed: int) -> torch.Tensor:
    """[FIELDS, members, N] m3/s on the device: gamma(0.8) fields of the given mean, each member with
    its own lognormal(0, 0.3) factor."""
    dev = _device()
    area = torch.as_tensor(host.map("grarea"), device=dev)
    with torch.random.fork_rng(devices=[dev]):
        torch.manual_seed(seed)
        shape = torch.full((FIELDS, area.numel()), 0.8, device=dev)
        field = torch.distributions.Gamma(shape, torch.full_like(shape, 0.8 / mean)).sample()
        factor = torch.exp(0.3 * torch.randn(members, device=dev) - 0.045).double()
    return (field.double() * area / 86_400_000.0)[:, None, :] * factor[:, None]


def _context(law: str, cells: int, members: int, seed: int, spinup: bool = True, **options):
    host, rivsto, mean = _network(law, cells)
    phys = PhysicsGPU(host, nmembers=members, **options)
    start = np.random.default_rng(seed).uniform(0.9, 1.1, (members, 1)) * rivsto
    phys.set_state({"rivsto": start})
    phys.calc_outpre()
    runoff = _runoff(host, mean, members, seed)
    torch.cuda.synchronize()
    if spinup:
        for h in range(SPINUP):
            phys.advance_device(1, runoff[h % FIELDS].data_ptr(), 0)
        phys.synchronize()
    return phys, runoff


def _pinned(shape) -> np.ndarray:
    return torch.zeros(shape, dtype=torch.float64).pin_memory().numpy()


def _host_fields(runoff: torch.Tensor) -> list:
    out = []
    for k in range(FIELDS):
        a = _pinned(tuple(runoff[k].shape))
        a[...] = runoff[k].cpu().numpy()
        out.append(a)
    return out


def _budgets(rows: list) -> np.ndarray:
    return np.array([[b[k] for k in sorted(b)] for b in rows])


# -------------------------------------------------------------------------------------- prepare
def prepare(case: dict, seed: int) -> dict:
    return globals()["_prepare_" + case["kind"]](case, seed) | {"kind": case["kind"], "hour": 0}


def _prepare_step(case, seed):
    phys, runoff = _context(case["law"], case["cells"], case["members"], seed)
    names = FULL_FIELDS if case.get("fields") == "full" else STEP_FIELDS
    return {"phys": phys, "runoff": _host_fields(runoff), "out": {n: _pinned(phys.diag_len(n)) for n in names}}


def _prepare_pipeline(case, seed):
    phys, runoff = _context(case["law"], case["cells"], case["members"], seed)
    outs = [{"outflw_aavg": _pinned(phys.M * phys.N)} for _ in range(2)]
    return {"phys": phys, "runoff": _host_fields(runoff), "outs": outs, "io": phys.pipeline(outs), "hours": case["hours"],
            "series": _pinned((case["hours"], phys.M * phys.N))}


def _prepare_ensemble(case, seed):
    phys, runoff = _context(case["law"], case["cells"], case["members"], seed)
    return {"phys": phys, "runoff": runoff, "view": E.Features(phys, np.ones(phys.N))}


def _prepare_batch(case, seed):
    weights = np.geomspace(1.0, 8.0, case["domains"])
    sizes = [max(2_000, int(case["cells"] * w / weights.sum())) for w in weights]
    parts = [_context(case["law"], n, case["members"], seed + 31 * d) for d, n in enumerate(sizes)]
    return {"ctx": [p for p, _ in parts], "runoff": [_host_fields(r) for _, r in parts],
            "out": [{"outflw_aavg": _pinned(p.M * p.N)} for p, _ in parts], "batch": PhysicsBatch([p for p, _ in parts])}


def _prepare_output(case, seed):
    phys, _ = _context(case["law"], case["cells"], case["members"], seed, ldiag_output=True)
    host = phys.host
    nxin, nyin, ix, iy, ia = synth.make_inpmat(host.nx, host.ny, host.i1seqx, host.i1seqy, host.map("grarea"), seed=1)
    phys.set_runoff_map((nxin, nyin, ix, iy, ia))
    phys.diag_output("reset")
    grids = np.random.default_rng(seed).gamma(0.8, 2.5, (FIELDS, phys.M, nyin, nxin)).astype(np.float32)
    return {"phys": phys, "grids": list(grids), "hours": case["hours"]}


def _mlp(seed: int, lr: float = 1e-3):
    mlp = E.MLP(_device(), seed=seed, lr=lr)
    weights = mlp.state_dict()
    rng = np.random.default_rng(seed)
    for k in range(3):
        weights["b"][k] = (0.1 * rng.standard_normal(weights["b"][k].shape)).astype(np.float32)
    weights["b"][3][0] = 0.7          # log1p of about the reference discharge
    mlp.load(weights)
    return mlp


def _prepare_emu_hour(case, seed):
    host, _, mean = _network(case["law"], case["cells"])
    plain, _ = _context(case["law"], case["cells"], 1, seed)
    mlp = _mlp(seed)
    mlp.residual = False              # the network predicts the hour's outflow itself
    ens = E.SurrogateEnsemble(host, mlp, members=case["members"], judge_slots=1, gauges=np.zeros(1, dtype=np.int64))
    for m in range(case["members"]):
        E.check(ens.lib.cmf_gpu_ctx_copy_member(ens.emu.h, m, plain.h, 0), "copy_member")
    plain.close()
    return {"ens": ens, "runoff": _runoff(host, mean, case["members"], seed), "input": ens.fe.runoff_view()}


def _rows(n: int, seed: int) -> torch.Tensor:
    g = torch.Generator(device=_device()).manual_seed(seed)
    x = torch.zeros(n, E.IN, dtype=torch.bfloat16, device=_device())
    for at in range(0, n, 1 << 20):
        part = x[at:at + (1 << 20)]
        part[:, :E.NFEAT] = torch.randn(part.shape[0], E.NFEAT, device=_device(), generator=g).to(torch.bfloat16)
    return x


def _prepare_infer(case, seed):
    return {"mlp": _mlp(seed), "x": _rows(case["rows"], seed), "y": torch.empty(case["rows"], device=_device())}


def _prepare_train(case, seed):
    g = torch.Generator(device=_device()).manual_seed(seed + 1)
    x = _rows(case["rows"], seed)
    target = 0.7 + 0.2 * x[:, 3].float() + 0.3 * torch.randn(case["rows"], device=_device(), generator=g)
    # the learning rate of the last steps of a training run (5 % of the first ones')
    return {"mlp": _mlp(seed, lr=5e-5), "x": x, "t": target.contiguous(), "valid": case["valid"]}


# ------------------------------------------------------------------------------------------ run
def run(state: dict):
    out = globals()["_run_" + state["kind"]](state)
    state["hour"] += 1
    return out


def _run_step(s):
    phys = s["phys"]
    phys.put_runoff(s["runoff"][s["hour"] % FIELDS])
    nt, dt, budgets = phys.advance()
    phys.get_diag_fields(s["out"])
    return {"nt": nt, "dt": dt, "budgets": _budgets(budgets), "fields": s["out"]}


def _run_pipeline(s):
    phys, io, n = s["phys"], s["io"], s["hours"]
    nts = np.zeros((n, phys.M), dtype=np.int32)
    at = s["hour"] * n
    phys.put_runoff_async(s["runoff"][at % FIELDS])
    io.advance()
    io.read_back(0)
    phys.put_runoff_async(s["runoff"][(at + 1) % FIELDS])
    io.advance()
    for k in range(n):
        nts[k] = io.wait()
        io.io_wait()
        s["series"][k] = s["outs"][k % 2]["outflw_aavg"]
        if k + 1 < n:
            io.read_back((k + 1) % 2)
        if k + 2 < n:
            phys.put_runoff_async(s["runoff"][(at + k + 2) % FIELDS])
            io.advance()
    return {"nt": nts, "discharge": s["series"]}


def _run_ensemble(s):
    s["phys"].advance_device(1, s["runoff"][s["hour"] % FIELDS].data_ptr(), 0)
    return {"discharge": s["view"].qprev(), "nt_dt": s["phys"].last_nt()}


def _run_batch(s):
    for phys, runoff in zip(s["ctx"], s["runoff"]):
        phys.put_runoff(runoff[s["hour"] % FIELDS])
    steps = s["batch"].advance()
    for phys, out in zip(s["ctx"], s["out"]):
        phys.get_diag_fields(out)
    return {"nt": [nt for nt, _, _ in steps], "dt": [dt for _, dt, _ in steps],
            "budgets": [_budgets(b) for _, _, b in steps], "fields": s["out"]}


def _run_output(s):
    phys, nts = s["phys"], []
    for k in range(s["hours"]):
        phys.put_runoff_grid(s["grids"][(s["hour"] + k) % FIELDS])
        nts.append(phys.advance()[0])
    phys.diag_output("getave")
    out = phys.get_diag_output()
    phys.diag_output("reset")
    return {"nt": nts, "output": out}


def _run_emu_hour(s):
    ens = s["ens"]
    s["input"].copy_(s["runoff"][s["hour"] % FIELDS])
    ens.emu_step()
    dt_min = ens.emu.stage()
    return {"discharge": ens.fe.qprev(), "dt_min": dt_min}


def _run_infer(s):
    return s["mlp"].infer_tc(s["x"], s["y"])


def _run_train(s):
    mlp = s["mlp"]
    loss = mlp.loss_and_grad(s["x"], s["t"], s["valid"])
    mlp.adam()
    return {"loss": loss, "gW": mlp.gW, "gb": mlp.gb, "W": mlp.W, "b": mlp.b}


# ----------------------------------------------------------------------------------------- work
def work(case: dict) -> dict:
    kind = case["kind"]
    net = E.NFEAT * E.HID + 2 * E.HID * E.HID + E.HID                       # weights the rows go through
    if kind == "infer":
        return {"bytes": case["rows"] * (2 * E.NFEAT + 4) + 2 * net, "flops": 2.0 * net * case["rows"]}
    if kind == "train":                                                     # forward, then both gradients
        return {"bytes": case["rows"] * (2 * E.NFEAT + 4) + 32 * net, "flops": 6.0 * net * case["rows"]}
    cells = case["cells"] * case["members"]
    if kind == "emu_hour":                                                  # state, runoff, maps in; state out
        return {"bytes": cells * 8 * (9 + 9 + 12), "flops": 2.0 * net * cells}
    hours = case.get("hours", 1)
    return {"bytes": float(cells) * hours * MEAN_NT * CELL_BYTES, "flops": float(cells) * hours * MEAN_NT * 300}


# ---------------------------------------------------------------------------------------- exact
def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind == "infer":
        return _exact_infer(prepare(case, seed))
    if kind == "train":
        return _exact_train(prepare(case, seed))
    if kind == "step" and case["law"] == "plain" and case.get("fields") != "full" and case["cells"] * case["members"] <= 300_000:
        s = prepare(case, seed)
        parts = [_exact_step(s["phys"], m, s["runoff"][0][m]) for m in range(case["members"])]
        return {"nt": None, "dt": np.array([p["dt"] for p in parts]), "budgets": np.stack([p["budgets"] for p in parts]),
                "fields": {n: np.concatenate([p[n] for p in parts]) for n in STEP_FIELDS}}
    return None      # channels, levees and dams: no short independent statement of them


def _exact_infer(s):
    w, b = [v.double() for v in s["mlp"].Wb], [v.double() for v in s["mlp"].b]
    out = torch.empty(s["x"].shape[0], dtype=torch.float64, device=_device())
    for at in range(0, out.numel(), 1 << 18):
        a = s["x"][at:at + (1 << 18)].double()
        for k in range(3):
            a = torch.relu(a @ w[k] + b[k])
        out[at:at + (1 << 18)] = a @ w[3][:, 0] + b[3][0]
    return out


def _exact_train(s):
    """Loss, gradients and Adam's first update of the network, products and sums in 64 bits."""
    mlp, n = s["mlp"], s["valid"]
    w = [v.double().requires_grad_() for v in mlp.Wb]
    b = [v.double().requires_grad_() for v in mlp.b]
    a = s["x"][:n].double()
    for k in range(3):
        a = torch.relu(a @ w[k] + b[k])
    y = (a @ w[3] + b[3])[:, 0]
    loss = ((y - s["t"][:n].double()) ** 2).sum() / n
    grads = torch.autograd.grad(loss, w + b)
    step = lambda p, g: p.double() - mlp.lr * g / (g.abs() + 1e-8)  # noqa: E731
    return {"loss": loss.detach(), "gW": list(grads[:4]), "gb": list(grads[4:]),
            "W": [step(p, g) for p, g in zip(mlp.W, grads[:4])], "b": [step(p, g) for p, g in zip(mlp.b, grads[4:])]}


def _exact_step(phys, m: int, runoff: np.ndarray) -> dict:
    """One coupling step of a plain network in numpy: stage scheme, CFL sub-steps, local-inertial
    outflow, outflow limiter, storage update."""
    host, prm = phys.host, phys.host.params
    n, layers = phys.N, phys.dims.nlfp
    mp = {k: host.map(k) for k in ("rivelv", "elevtn", "nxtdst", "rivwth", "rivhgt", "rivlen", "rivman", "grarea",
                                   "rivstomax", "dwnelv", "i2mask")}
    smax, grad = host.map("fldstomax").reshape(layers, n), host.map("fldgrd").reshape(layers, n)
    nxt = host.map("i1next") - 1
    river = nxt >= 0
    down = np.where(river, nxt, 0)
    length, width, rsm = mp["rivlen"], mp["rivwth"], mp["rivstomax"]
    dst = np.where(river, mp["nxtdst"], prm.pdstmth)
    inc = mp["grarea"] / length * prm.dfrcinc
    f32 = lambda v: float(np.float32(v))  # noqa: E731

    def stage(total):
        full = (total[None] > smax).cumprod(0).astype(bool)
        cnt = full.sum(0)
        sfil, dfil = rsm.copy(), np.zeros(n)
        for k in range(layers):
            sfil = np.where(full[k], smax[k], sfil)
            dfil = np.where(full[k], dfil + grad[k] * inc, dfil)
        wfil = width + cnt * inc
        over = cnt >= layers
        g = grad[np.minimum(cnt, layers - 1), np.arange(n)]
        with np.errstate(invalid="ignore"):
            wadd = np.where(over, 0.0, -wfil + np.sqrt(wfil * wfil + 2.0 * (total - sfil) / length / g))
        fld = np.where(over, dfil + (total - sfil) / wfil / length, dfil + g * wadd)
        wet = total > rsm
        riv = np.where(wet, np.minimum(rsm + length * width * fld, total), total)
        frac = np.clip((-width + wfil + wadd) / (inc * layers), 0.0, 1.0)
        return (riv, np.maximum(total - riv, 0.0) * wet, np.maximum(riv / length / width, 0.0), np.where(wet, fld, 0.0),
                np.where(wet, frac, 0.0))

    def gather(v):                     # sum over upstream cells, ascending
        return np.bincount(nxt[river], weights=v[river], minlength=n)

    st = {k: v[m] for k, v in phys.get_state().items() if v.shape[1] == n}
    riv, fld, dph, fdph, frac = stage(st["rivsto"] + st["fldsto"])
    rpre, fpre, dpre, spre = st["rivout_pre"], st["fldout_pre"], st["rivdph_pre"], st["fldsto_pre"]
    ddph = np.maximum(dph, 0.01)
    dt_def = host.dt
    dt_min = min(dt_def, float(np.min((prm.pcadp * dst * (prm.pgrv * ddph) ** -0.5)[mp["i2mask"] == 0])))
    nt = int(dt_def / dt_min - f32(0.01)) + 1
    dt = dt_def * float(np.float32(1.0) / np.float32(nt))
    elv, bank = mp["rivelv"], mp["elevtn"]
    flow_sum = np.zeros(n)
    for _ in range(nt):
        sfc, sfc_pre = elv + dph, elv + dpre
        low = np.where(river, sfc[down], mp["dwnelv"])
        low_pre = np.where(river, sfc_pre[down], -np.inf)
        top, top_pre = np.where(river, np.maximum(sfc, low), sfc), np.maximum(sfc_pre, low_pre)
        slope = (sfc - low) / dst
        deep, deep_pre = top - elv, top_pre - elv
        im = np.maximum(np.sqrt(np.maximum(deep * deep_pre, 0.0)), 1e-6)
        area = np.maximum(width * deep, 1e-10)
        q0 = rpre / width
        gdt = prm.pgrv * dt
        rout = width * (q0 + gdt * im * slope) / (1.0 + gdt * mp["rivman"] ** 2 * np.abs(q0) * im ** (-7.0 / 3.0))
        rout = np.where((im > f32(1e-5)) & (area > f32(1e-5)), rout, 0.0)
        farea = np.maximum(fld / length - fdph * width, 0.0)
        fdeep, fdeep_pre = np.maximum(top - bank, 0.0), top_pre - bank
        fim = np.maximum(np.sqrt(np.maximum(fdeep * fdeep_pre, 0.0)), 1e-6)
        farea_pre = np.maximum(spre / length - np.maximum(dpre - mp["rivhgt"], 0.0) * width, 1e-6)
        aim = np.maximum(np.sqrt(farea * farea_pre), 1e-6)
        fout = (fpre + gdt * aim * np.clip(slope, -0.005, 0.005)) / (
            1.0 + gdt * prm.pmanfld ** 2 * np.abs(fpre) * fim ** (-4.0 / 3.0) / aim)
        fout = np.where((fim > 1e-5) & (farea > 1e-5), fout, 0.0)
        fout = np.where(fout * rout > 0.0, fout, 0.0)
        limit = np.minimum(0.05 * (riv + fld) / np.maximum((-rout - fout) * dt, f32(1e-10)), 1.0)
        limit = np.where(river, limit, 1.0)
        rout, fout = rout * limit, fout * limit
        need = (np.maximum(rout, 0.0) + np.maximum(fout, 0.0) + gather(np.maximum(-rout, 0.0) + np.maximum(-fout, 0.0))) * dt
        rate = np.minimum((riv + fld) / np.maximum(need, 1e-10), 1.0)
        by = np.where((rout > 0.0) | ~river, rate, rate[down])
        rout, fout = rout * by, fout * by
        rinf, finf = gather(rout), gather(fout)
        pre = riv + fld
        r = riv + rinf * dt - rout * dt
        f = np.where(r < 0.0, fld + r, fld)
        r = np.maximum(r, 0.0)
        f = f + finf * dt - fout * dt
        r = np.where(f < 0.0, np.maximum(r + f, 0.0), r)
        f = np.maximum(f, 0.0)
        after = r + f
        r, f = r + runoff * (1.0 - frac) * dt, f + runoff * frac * dt
        rpre, fpre, dpre, spre = rout, fout, dph, fld
        riv, fld, dph, fdph, frac = stage(r + f)
        flow_sum += (rout + fout) * dt
    b = {"stopre": pre.sum(), "stonxt": after.sum(), "stonew": (r + f).sum(), "rivinf": ((rinf + finf) * dt).sum(),
         "rivout": ((rout + fout) * dt).sum(), "stopre2": (r + f).sum(), "stonew2": (riv + fld).sum(), "rivsto": riv.sum(),
         "fldsto": fld.sum(), "fldare": (mp["grarea"] * frac).sum(), "levsto": 0.0, "dam_miss": 0.0}
    return {"dt": dt, "budgets": np.array([b[k] for k in sorted(b)]), "outflw_aavg": flow_sum / (nt * dt), "rivdph": dph,
            "storge": riv + fld}
