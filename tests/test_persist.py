"""The persistent schedule (launch_mode 2): one cooperative kernel per coupling step with grid
barriers between the phases and the cell tiles interleaved over the CTAs.

It runs the same per-cell arithmetic as the graph of phase kernels, so states, NT/DT and budgets
must equal that path bit for bit (the budgets with the same 256-cell partial blocks), and the oracle
within the parity tolerance.  Its bounded waits are checked by a barrier that cannot complete."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import rel_close, runoff_series
from cmf_b200 import synth

pytestmark = pytest.mark.gpu

RTOL = 1e-9
STATE_KEYS = ("rivsto", "fldsto", "rivout", "fldout", "rivout_pre", "fldout_pre", "rivdph_pre", "fldsto_pre",
              "levsto", "damsto", "daminf", "pthflw")
DIAG_KEYS = ("rivdph", "flddph", "fldfrc", "fldare", "sfcelv", "storge", "rivvel", "rivinf", "fldinf", "pthout",
             "outflw", "pthflwsum", "levdph", "rivout_aavg", "fldout_aavg", "outflw_aavg", "rivvel_aavg",
             "pthout_aavg", "runoff_aavg", "daminf_aavg", "storge_amax", "outflw_amax", "rivdph_amax",
             "pthflw_aavg", "pthflwsum_aavg")


def _same(a, b):
    return np.array_equal(np.ascontiguousarray(a).view(np.int64), np.ascontiguousarray(b).view(np.int64))


@pytest.mark.parametrize("name,members,nsteps", [("stress", 1, 30), ("cfg1s", 3, 16), ("cfg0", 2, 30)])
def test_persistent_equals_graph_bit_for_bit(case_dirs, name, members, nsteps):
    """Every state and diagnostic array, NT, DT and the budgets of every step are bit-identical to
    the graph of phase kernels (block size 256, the persistent kernel's tile)."""
    from cmf_b200 import HostModel, PhysicsGPU

    h = HostModel(case_dirs[name])
    a = PhysicsGPU(h, nmembers=members, launch_mode=2, ldiag_output=True)
    b = PhysicsGPU(h, nmembers=members, launch_mode=0, block_size=256, ldiag_output=True)
    assert a.launch_mode == 2 and b.launch_mode == 0
    gr = h.map("grarea")
    series = [list(runoff_series(gr, name, nsteps, seed=s, hourly=(name != "cfg0"))) for s in range(members)]
    for k in range(nsteps):
        r = np.stack([series[m][k] for m in range(members)])
        a.put_runoff(r)
        b.put_runoff(r)
        na, da, ba = a.advance()
        nb, db, bb = b.advance()
        assert np.array_equal(na, nb) and _same(da, db), f"step {k}: NT/DT"
        for m in range(members):
            for f, v in ba[m].items():
                assert _same(np.float64(v), np.float64(bb[m][f])), f"step {k} member {m} budget {f}"
        if k == nsteps // 2:
            a.diag_output("getave")
            b.diag_output("getave")
            oa, ob = a.get_diag_output(), b.get_diag_output()
            for f in oa:
                assert _same(oa[f], ob[f]), f"output diagnostics {f}"
            a.diag_output("reset")
            b.diag_output("reset")
    sa, sb = a.get_state(), b.get_state()
    for f in STATE_KEYS:
        assert _same(sa[f], sb[f]), f
    ga, gb = a.get_diag(), b.get_diag()
    for f in DIAG_KEYS:
        assert _same(ga[f], gb[f]), f
    assert a.kernel_launches < b.kernel_launches


# (scale of the config-1 grid, members, path levels): a net of a few cells in its last tile, more members
# than a group holds, paths of more levels than a warp has lanes, 23 tasks per SM (the form with more
# registers) and 25 (the other), two groups of a large member, and a member that does not
# fit the SMs (the kernel over global memory)
@pytest.mark.parametrize("scale,members,levels", [(0.012, 1, 5), (0.012, 70, 33), (0.05, 1, 64), (0.1, 29, 5), (0.1, 30, 5),
                                                  (0.6, 4, 3), (1.05, 1, 5)])
def test_resident_edges_equal_graph_bit_for_bit(tmp_path, scale, members, levels):
    """Three flooded steps of nets at the edges of the resident kernel's tiles, groups and register forms
    leave the same bits as the graph of phase kernels."""
    from cmf_b200 import HostModel, PhysicsGPU

    spec = synth.spec_config1(seed=3, scale=scale)
    spec.npthlev = levels
    spec.rivhgt_scale = 0.3
    synth.write_case(synth.make_case(spec), str(tmp_path / "c"))
    h = HostModel(str(tmp_path / "c"))
    series = np.stack(list(runoff_series(h.map("grarea"), "stress", 3, hourly=True)))
    weight = np.random.default_rng(2).uniform(0.5, 2.0, (members, 1))
    a = PhysicsGPU(h, nmembers=members, launch_mode=2, ldiag_output=True)
    b = PhysicsGPU(h, nmembers=members, launch_mode=0, block_size=256, ldiag_output=True)
    for r in series:
        steps = []
        for g in (a, b):
            g.put_runoff(weight * r)
            steps.append(g.advance())
        (na, da, ba), (nb, db, bb) = steps
        assert np.array_equal(na, nb) and _same(da, db)
        for m in range(members):
            assert all(_same(np.float64(v), np.float64(bb[m][f])) for f, v in ba[m].items()), m
    sa, sb = a.get_state(), b.get_state()
    ga, gb = a.get_diag(), b.get_diag()
    for f in STATE_KEYS:
        assert _same(sa[f], sb[f]), f
    for f in DIAG_KEYS:
        assert _same(ga[f], gb[f]), f


def test_persistent_vs_oracle(case_dirs):
    """Free-running parity of the persistent schedule against the oracle on config-1 laws (levees,
    dams, bifurcation channels), 48 hourly steps."""
    from cmf_b200 import HostModel, PhysicsGPU
    from oracle import Oracle

    h = HostModel(case_dirs["cfg1s"])
    g = PhysicsGPU(h, launch_mode=2)
    o = Oracle(case_dirs["cfg1s"])
    for k, r in enumerate(runoff_series(h.map("grarea"), "cfg1s", 48, hourly=True)):
        o.put_runoff(r)
        g.put_runoff(r)
        nt_o, dt_o = o.advance()
        nt_g, dt_g, _ = g.advance()
        assert nt_g[0] == nt_o and dt_g[0] == dt_o, f"step {k}"
    st = g.get_state()
    for f in ("rivsto", "fldsto", "rivout", "fldout", "levsto", "damsto", "pthflw"):
        ok, worst, bad = rel_close(st[f][0], o.d(f), RTOL)
        assert ok, (f, worst, bad)


def test_persistent_bounded_wait_returns_status(case_dirs):
    """A grid barrier that can never complete (its count is one arrival short) runs out its 2 ms
    bound on every CTA: the kernel returns, the host reads CMF_E_BARRIER, and the context then
    advances normally, equal to a context that never ran the check."""
    from cmf_b200 import HostModel, PhysicsGPU

    h = HostModel(case_dirs["cfg1s"])
    g = PhysicsGPU(h, launch_mode=2)
    ref = PhysicsGPU(h, launch_mode=2)
    series = list(runoff_series(h.map("grarea"), "cfg1s", 6, hourly=True))
    g.put_runoff(series[0])
    ref.put_runoff(series[0])
    g.advance()
    ref.advance()
    assert g.persist_selftest(2_000_000) == 5
    for r in series[1:]:
        g.put_runoff(r)
        ref.put_runoff(r)
        a, _, _ = g.advance()
        b, _, _ = ref.advance()
        assert a[0] == b[0]
    sa, sb = g.get_state(), ref.get_state()
    for f in ("rivsto", "fldsto", "rivout", "fldout"):
        assert _same(sa[f], sb[f]), f


@pytest.mark.parametrize("scale", [None, 1.05])
@pytest.mark.parametrize("read", ["last_nt", "advance"])
def test_step_after_an_aborted_one_takes_its_own_minimum(case_dirs, tmp_path, scale, read):
    """A step that gives up at its first grid barrier has merged its cells' CFL minima.  The call that
    reads the control blocks reports CMF_E_BARRIER, and a step from a new state then takes NT and DT
    from that state alone (resident kernel, and the one over global memory)."""
    from cmf_b200 import HostModel, PhysicsGPU

    d = case_dirs["cfg1s"]
    if scale:
        d = str(tmp_path / "c")
        synth.write_case(synth.make_case(synth.spec_config1(seed=3, scale=scale)), d)
    h = HostModel(d)
    g, ref = PhysicsGPU(h, launch_mode=2), PhysicsGPU(h, launch_mode=2)
    r = next(iter(runoff_series(h.map("grarea"), "cfg1s", 1)))
    g.put_runoff(r)
    ref.put_runoff(r)
    deep, _, _ = g.advance()
    g.persist_selftest_step(2_000_000)
    with pytest.raises(Exception, match="barrier"):
        getattr(g, read)()
    shallow = h.initial_state()
    shallow["rivsto"] = 1e-3 * shallow["rivsto"]
    for p in (g, ref):
        p.set_state(shallow)
    nt, dt, _ = g.advance()
    nt_ref, dt_ref, _ = ref.advance()
    assert nt_ref[0] < deep[0]
    assert nt[0] == nt_ref[0] and _same(dt, dt_ref)
    sa, sb = g.get_state(), ref.get_state()
    for f in STATE_KEYS:
        assert _same(sa[f], sb[f]), f


def test_resident_buffers_are_made_on_first_use(case_dirs):
    """Contexts whose schedule is one of phase kernels hold none of the resident kernel's buffers (budget
    terms alone are 96 B per cell and member); they appear when a schedule first runs it."""
    import torch

    from cmf_b200 import HostModel, PhysicsGPU

    h = HostModel(case_dirs["cfg1s"])
    M, N = 64, h.dims.nseqall
    need = 96 * M * N
    free = lambda: torch.cuda.mem_get_info(0)[0]  # noqa: E731

    def made(**kw):
        torch.cuda.synchronize()
        before = free()
        p = PhysicsGPU(h, nmembers=M, **kw)
        return p, before - free()

    made(launch_mode=2)[0].close()               # modules and streams of a first context
    resident, with_buffers = made(launch_mode=2)
    resident.close()
    for kw in (dict(launch_mode=1), dict(block_size=128)):
        p, bytes_ = made(**kw)
        assert bytes_ <= with_buffers - need, (kw, bytes_, with_buffers, need)
        if "block_size" in kw:
            at = free()
            p.set_schedule(mode=2)
            assert at - free() >= need
            p.put_runoff(np.zeros((M, N)))
            p.advance()
        p.close()


@pytest.mark.parametrize("upstream", [15, 16, 40])
def test_persistent_with_many_upstream_cells(case_dirs, upstream):
    """A cell of 15 upstream cells is the widest the resident kernel packs; with more the persistent
    schedule runs the kernel over global memory.  Both leave the bits of the graph of phase kernels."""
    import ctypes as C

    from cmf_b200 import HostModel, PhysicsGPU

    h = HostModel(case_dirs["cfg1s"])
    N, R = h.dims.nseqall, h.dims.nseqriv
    nxt = np.ctypeslib.as_array(h.maps.i1next, shape=(N,))
    # headwaters of plain channels drain into the last river cell but a few
    target = R - 5
    dam, mask = h.map("i1dam"), h.map("i2mask")
    heads = [i for i in range(target) if not np.any(nxt[:R] == i + 1) and dam[i] == 0 and mask[i] == 0 and nxt[i] != target + 1]
    have = int((nxt[:R] == target + 1).sum())
    for i in heads[:upstream - have]:
        nxt[i] = target + 1
    lists = [np.flatnonzero(nxt[:R] == j + 1) + 1 for j in range(N)]
    most = max(len(v) for v in lists)
    assert most == upstream
    upst = np.zeros((most, N), dtype=np.int32)
    upn = np.array([len(v) for v in lists], dtype=np.int32)
    for j, v in enumerate(lists):
        upst[:len(v), j] = v
    h.dims.upnmax = most
    h.maps.i1upst = upst.ctypes.data_as(C.POINTER(C.c_int32))
    h.maps.i1upn = upn.ctypes.data_as(C.POINTER(C.c_int32))
    series = list(runoff_series(h.map("grarea"), "stress", 4, hourly=True))
    a = PhysicsGPU(h, nmembers=2, launch_mode=2)
    b = PhysicsGPU(h, nmembers=2, launch_mode=0, block_size=256)
    for r in series:
        for p in (a, b):
            p.put_runoff(np.stack([r, 2.0 * r]))
        (na, da, ba), (nb, db, bb) = a.advance(), b.advance()
        assert np.array_equal(na, nb) and _same(da, db) and ba == bb
    sa, sb = a.get_state(), b.get_state()
    ga, gb = a.get_diag(), b.get_diag()
    for f in STATE_KEYS:
        assert _same(sa[f], sb[f]), f
    for f in DIAG_KEYS:
        assert _same(ga[f], gb[f]), f


def test_member_state_takes_its_arrays_and_no_more(case_dirs):
    """The device memory a member adds is that of its arrays (332 B per cell with diagnostics, levees and
    dams, and its paths' 144 B each), not of 60 allocations rounded up."""
    import torch

    from cmf_b200 import HostModel, PhysicsGPU

    h = HostModel(case_dirs["cfg1s"])
    N, P = h.dims.nseqall, h.dims.npthout
    assert h.dims.npthlev == 5

    def made(members):
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info(0)[0]
        p = PhysicsGPU(h, nmembers=members, block_size=128)
        torch.cuda.synchronize()
        used = before - torch.cuda.mem_get_info(0)[0]
        p.close()
        return used

    made(1)                                      # modules and streams of a first context
    assert made(64) - made(1) <= 63 * (332 * N + 144 * P) + 8 * 2 ** 20
