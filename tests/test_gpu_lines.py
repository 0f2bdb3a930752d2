"""The line kernels of the explicit stage at the sizes where a warp's share of
a line ends: i lines of 30 / 31 cells and faces per warp, 32 lanes along i,
segments of a few faces, lines of two cells, more norm rows than one CTA sums,
and a store schedule that needs several groups of blocks."""
import numpy as np
import pytest

import casekit
from cosa_b200 import cases, gpu

pytestmark = pytest.mark.gpu


def _run(case, q, metrics, schedule, ncyc):
    ctx = gpu.Context([case.tables], case.params)
    m = [ctx.alloc_p2().upload(a) for a in metrics]
    d = ctx.alloc_p3().upload(q)
    ctx.bind_level(1, q=d, qold=ctx.alloc_p3(), dtvol=ctx.alloc_p1(), si=m[0], sj=m[1], sk=m[2])
    ctx.set_schedule(1, schedule)
    hist, st = ctx.smooth(1, ncyc, 1, 1)
    assert st == 0
    out = d.download()
    ctx.close()
    return out, hist


@pytest.mark.parametrize("dims", [(2, 2, 2), (29, 3, 2), (30, 5, 2), (31, 16, 3), (32, 17, 2), (33, 4, 5), (61, 33, 2),
                                  (64, 64, 40)])
def test_line_kernels_at_their_edges(oracle_mod, dims):
    """Both schedules against the oracle (1e-12 of each variable's scale, the
    bound of the other FP64 parity tests) and, bit for bit, each other."""
    case = cases.bump_channel(*dims, kface_bc=80)
    O = oracle_mod.OracleLevel(case.tables, case.params)
    si, sj, sk, _ = O.metrics(case.x, case.y, case.z)
    q = cases.perturbed_state(case, amp=0.01, seed=sum(dims))
    qo = q.copy()
    ncyc = 1 if dims[2] > 8 else 2
    hist_o, st = O.smooth(qo, si, sj, sk, ncyc, rms_every=1)
    assert st == 0
    res = [_run(case, q, (si, sj, sk), s, ncyc) for s in (0, 1)]
    a, b = (casekit.interior_cells(case, r[0], 5) for r in res)
    assert np.array_equal(a, b)
    o = casekit.interior_cells(case, qo, 5)
    sc = np.abs(o).reshape(-1, 5).max(axis=0)
    sc[1:4] = sc[1:4].max()
    assert (np.abs(a - o) / sc[None, :, None]).max() <= 1e-12
    for _, h in res:
        np.testing.assert_allclose(h, hist_o, rtol=1e-9)


def test_store_schedule_in_groups_equals_chain():
    """4.2 M cells in 24 blocks: the store schedule's flux buffer holds a part
    of the blocks at a time."""
    case = cases.duct3d(segs=[[72, 88], [32, 40, 64], [64, 48, 48, 32]])
    ctx = gpu.Context([case.tables], case.params)
    X, Y, Z = (ctx.alloc_p2(ncomp=1).upload(a) for a in (case.x, case.y, case.z))
    si, sj, sk = (ctx.alloc_p2() for _ in range(3))
    ctx.imetrix(1, X, Y, Z, si, sj, sk)
    q = ctx.alloc_p3()
    ctx.bind_level(1, q=q, qold=ctx.alloc_p3(), dtvol=ctx.alloc_p1(), si=si, sj=sj, sk=sk)
    out = []
    for schedule in (0, 1):
        q.upload(case.q0)
        ctx.set_schedule(1, schedule)
        _, st = ctx.smooth(1, 2, 1, 1)
        assert st == 0
        out.append(q.download())
    ctx.close()
    assert np.array_equal(out[0], out[1])


@pytest.mark.parametrize("irsop", [1, 3])
@pytest.mark.parametrize("ni", [3, 31, 33, 450, 900, 1700, 3300])
def test_irs_line_lengths(oracle_mod, ni, irsop):
    """Residual smoothing of lines that fit shared memory 32, 16 or 8 at a time
    and (1700 varying, 3300) do not: cirs against the oracle, and one fused
    cycle, which scales in the sweeps where it can."""
    case = cases.bump_channel(ni, 6, 2)
    p = case.params
    p.irsop, p.psirs, p.rat = irsop, 0.125, float(np.sqrt(1 + 4 * 0.6))
    O = oracle_mod.OracleLevel(case.tables, p)
    si, sj, sk, _ = O.metrics(case.x, case.y, case.z)
    q = cases.perturbed_state(case, amp=0.01, seed=ni)
    res, dt, _ = O.residual(q.copy(), si, sj, sk)
    lam, qp = O.p3(), q.copy()
    O.cons2prim(qp)
    O.lambda_(qp, si, sj, sk, lam)
    beta = [O.p1() for _ in range(3)]
    O.deltat(dt, lam, *beta)
    ctx = gpu.Context([case.tables], p)
    rg = ctx.alloc_p3().upload(res)
    ctx.cirs(1, rg, ctx.alloc_p1().upload(dt), *(ctx.alloc_p1().upload(a) for a in beta))
    oracle_mod.irs(O, res, dt, *beta)

    def off(a, b):
        a, b = (casekit.interior_cells(case, x, 5) for x in (a, b))
        sc = np.abs(b).reshape(-1, 5).max(axis=0)
        sc[1:4] = sc[1:4].max()
        return (np.abs(a - b) / sc[None, :, None]).max()

    assert off(rg.download(), res) <= 1e-12
    qo = q.copy()
    _, st, _, _ = oracle_mod.smooth_irs(O, qo, si, sj, sk, 1, rms_every=1)
    assert st == 0
    m = [ctx.alloc_p2().upload(a) for a in (si, sj, sk)]
    d = ctx.alloc_p3().upload(q)
    ctx.bind_level(1, q=d, qold=ctx.alloc_p3(), dtvol=ctx.alloc_p1(), si=m[0], sj=m[1], sk=m[2],
                   betaxi=ctx.alloc_p1(), betaeta=ctx.alloc_p1(), betazeta=ctx.alloc_p1())
    _, st = ctx.smooth(1, 1, 1, 1)
    assert st == 0
    assert off(d.download(), qo) <= 1e-12
    ctx.close()
