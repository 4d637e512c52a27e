"""The element-mode batch kernel (rve_modes_kernel.cuh) at the edges of its
range: warps whose rows start at lane 0 or straddle warps, one and two planes
per half, odd and even plane counts, the largest meshes of each kernel class,
two and three strips of rows, 32 element layers, and the first meshes past the
range (which keep the block-stencil kernel), cubic and box elements, all in
one batch.

Solves run to a relative residual of 1e-10; a stress error above 1e-8 of
max|stress| (the suite's tolerance for a 1e-8 residual) is a wrong operator,
not a stopping error."""
import ctypes as C

import numpy as np
import pytest

import madmax_b200 as mb
from oracle import oracle as O

pytestmark = pytest.mark.gpu

MESHES = [(2, 2, 2), (2, 3, 4), (3, 2, 5), (4, 4, 3), (8, 8, 5), (8, 4, 9), (9, 9, 4), (10, 7, 6),
          (12, 12, 3), (16, 16, 4), (16, 10, 7), (32, 3, 4), (31, 4, 3), (20, 20, 3), (13, 31, 2),
          (25, 25, 3), (26, 25, 3), (5, 4, 31), (5, 4, 32), (5, 4, 33),
          (31, 33, 2), (32, 32, 3), (33, 31, 2), (33, 32, 2)]


def voxel_batch(cube, seed):
    rng = np.random.default_rng(seed)
    descs, ets, meshes = [], [], []
    for n in MESHES:
        edge = rng.uniform(0.05, 0.2, 3)
        # cubes: edges of exactly 1/8
        ln = [n[k] / 8.0 if cube else n[k] * edge[k] for k in range(3)]
        d = mb.rve_desc(n, 0.2, (1e9, 1e9 * float(np.exp(rng.uniform(np.log(2), np.log(100))))),
                        (float(rng.uniform(0.2, 0.35)), float(rng.uniform(0.2, 0.35))), ln)
        descs.append(d)
        ets.append((rng.random(n[0] * n[1] * n[2]) < 0.4).astype(np.uint8))
        meshes.append(O.mesh(3, [v + 1 for v in n], ln))
    return descs, ets, meshes, rng.normal(0, 1e-3, (len(MESHES), 3, 6))


@pytest.mark.parametrize("cube", [True, False])
@pytest.mark.parametrize("precision", [mb.SP_PREC_MIXED, mb.SP_PREC_FP64])
def test_edges_match_oracle(precision, cube):
    descs, ets, meshes, eps = voxel_batch(cube, 5 + cube)
    b = mb.Batch(descs, nrhs=3, rtol=1e-10, threads=512, ctas_per_sm=1, precision=precision)
    for i, et in enumerate(ets):
        b.set_etype(i, et)
    stress, strain, info = b.homogenize(np.ascontiguousarray(eps))
    inf = mb.info_array(info)
    assert (inf["status"] == 0).all() and (inf["relres"] <= 1e-10).all()
    assert b.last_launches() > 2
    for i, d in enumerate(descs):
        _, st, _, _ = O.homogenize(meshes[i], ets[i], tuple(d.E), tuple(d.nu), eps[i], rtol=1e-12,
                                   lin_rtol=1e-13)
        assert np.abs(stress[i] - st).max() <= 1e-8 * np.abs(st).max(), (MESHES[i], cube)
        assert np.allclose(strain[i], eps[i], rtol=0, atol=1e-15), MESHES[i]


@pytest.mark.parametrize("periodic", [False, True])
def test_one_warp_launch(periodic):
    """A launch whose largest RVE needs one warp (the tables are filled by as
    few threads), affine and periodic, against the oracles."""
    from oracle import periodic as PER
    d = mb.rve_desc(4, 0.3, (1e9, 3e10), (0.31, 0.22))
    s, _, info = mb.Batch([d], rtol=1e-10, threads=512, ctas_per_sm=1,
                          bc=mb.SP_BC_PERIODIC if periodic else mb.SP_BC_AFFINE).homogenize()
    m = O.cube_mesh(4)
    et = O.fiber_types(m, [1, 1], d.radius)
    if periodic:
        _, st, _ = PER.homogenize_periodic(m, et, tuple(d.E), tuple(d.nu), np.eye(6))
    else:
        _, st, _, _ = O.homogenize(m, et, tuple(d.E), tuple(d.nu), np.eye(6), rtol=1e-12,
                                   lin_rtol=1e-13)
    assert info[0].status == 0
    assert np.abs(s[0] - st).max() <= 1e-8 * np.abs(st).max()


PER_MESHES = [(2, 2, 2), (3, 2, 3), (2, 5, 4), (7, 7, 5), (15, 4, 6), (8, 8, 7), (31, 3, 2),
              (17, 17, 3), (4, 3, 30), (4, 3, 31), (24, 24, 2), (25, 25, 2)]


@pytest.mark.parametrize("cube", [True, False])
def test_periodic_edges_match_fp64(cube):
    """Periodic conditions: rows that start at lane 0 or straddle warps, odd
    and even plane counts (the halves' seams), 30 and 31 layers, the largest
    classes, on random voxel materials; against the FP64 periodic batch (which
    is tested against the periodic oracle), both solved to 1e-10."""
    rng = np.random.default_rng(41 + cube)
    descs, ets = [], []
    for n in PER_MESHES:
        edge = rng.uniform(0.05, 0.2, 3)
        ln = [n[k] / 8.0 if cube else n[k] * edge[k] for k in range(3)]
        descs.append(mb.rve_desc(n, 0.2, (1e9, 1e9 * float(rng.uniform(2, 100))), (0.3, 0.25), ln))
        ets.append((rng.random(n[0] * n[1] * n[2]) < 0.4).astype(np.uint8))
    eps = rng.normal(0, 1e-3, (len(descs), 3, 6))
    out = []
    for kw in ({"threads": 512, "ctas_per_sm": 1}, {"precision": mb.SP_PREC_FP64, "threads": 512,
                                                    "ctas_per_sm": 2}):
        b = mb.Batch(descs, nrhs=3, rtol=1e-10, bc=mb.SP_BC_PERIODIC, **kw)
        for i, et in enumerate(ets):
            b.set_etype(i, et)
        s, strain, info = b.homogenize(np.ascontiguousarray(eps))
        assert (mb.info_array(info)["status"] == 0).all()
        assert np.allclose(strain, eps, rtol=0, atol=1e-14)
        out.append(s)
    for i in range(len(descs)):
        assert np.abs(out[0][i] - out[1][i]).max() <= 1e-8 * np.abs(out[1][i]).max(), PER_MESHES[i]


def test_trivial_load_cases():
    """A zero strain gives zero stress, and a homogeneous RVE is solved by the
    affine start: no CG iteration, stress = D strain."""
    descs = [mb.rve_desc(n, 0.3, (2e9, 2e9), (0.3, 0.3)) for n in (2, 5, 16, 21)]
    eps = np.zeros((len(descs), 2, 6))
    eps[:, 1] = np.random.default_rng(3).normal(0, 1e-3, (len(descs), 6))
    s, _, info = mb.Batch(descs, nrhs=2, threads=512, ctas_per_sm=1).homogenize(eps)
    inf = mb.info_array(info)
    assert (inf["status"] == 0).all() and (inf["inner"] == 0).all()
    D = np.zeros(36)
    O.lib().orc_iso_D(3, 2e9, 0.3, O.ptr(D))
    for i in range(len(descs)):
        assert (s[i, 0] == 0).all()
        ref = D.reshape(6, 6) @ eps[i, 1]
        assert np.abs(s[i, 1] - ref).max() <= 1e-12 * np.abs(ref).max()


def test_parallel_launches_captured_in_a_graph():
    """A batch of several kernel classes launches them on parallel streams;
    captured in a CUDA graph and replayed, it gives the direct launch's
    results bit for bit."""
    import torch
    rng = np.random.default_rng(8)
    descs = [mb.rve_desc(int(n), float(rng.uniform(0.1, 0.35)), (1e9, 2e10), (0.3, 0.2))
             for n in (6, 12, 20, 24, 33, 16, 9, 6)]
    b = mb.Batch(descs, threads=512, ctas_per_sm=1)
    s = torch.cuda.Stream()
    sp = C.c_void_p(s.cuda_stream)
    direct, out = np.zeros((len(descs), 6, 6)), np.zeros((len(descs), 6, 6))
    b.launch(sp)
    b.download(direct, None, None, sp)
    s.synchronize()
    assert b.last_launches() == 6
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        b.launch(sp)
    for _ in range(2):
        out[:] = 0
        info = (mb.sp_solve_info * len(descs))()
        g.replay()
        torch.cuda.synchronize()
        b.download(out, None, info, sp)
        s.synchronize()
        assert (mb.info_array(info)["status"] == 0).all()
        assert np.array_equal(out, direct)
    del g
    b.close()


@pytest.mark.parametrize("length,E,strain", [(1.0, 1e9, 1e-14), (1.0, 1e9, 1e-18),
                                             (1e-6, 1e9, 1e-6), (1e-6, 1e9, 1e-10),
                                             (1e-9, 1.0, 1e-3)])
@pytest.mark.parametrize("periodic", [False, True])
def test_units_do_not_matter(periodic, length, E, strain):
    """Small strains, lengths and moduli: the squared residuals that steer the
    FP32 corrections are far below the smallest FP32 number.  The stress of a
    linear RVE scales with E and the strain and not with its size, so the
    oracle solves the RVE of unit length."""
    from oracle import periodic as PER
    rng = np.random.default_rng(31)
    meshes = [(4, 4, 4), (7, 5, 6), (8, 8, 5)] if periodic else [(4, 4, 4), (7, 5, 6), (17, 24, 7)]
    descs, ets, refs = [], [], []
    eps = rng.normal(0, 1.0, (len(meshes), 2, 6))
    for i, n in enumerate(meshes):
        ln = [v / 8.0 for v in n]
        nu = (0.3, 0.22)
        descs.append(mb.rve_desc(n, 0.2, (E, 30 * E), nu, [v * length for v in ln]))
        ets.append((rng.random(n[0] * n[1] * n[2]) < 0.4).astype(np.uint8))
        m = O.mesh(3, [v + 1 for v in n], ln)
        if periodic:
            st = PER.homogenize_periodic(m, ets[i], (1.0, 30.0), nu, eps[i])[1]
        else:
            st = O.homogenize(m, ets[i], (1.0, 30.0), nu, eps[i], rtol=1e-12, lin_rtol=1e-13)[1]
        refs.append(np.asarray(st) * E * strain)
    b = mb.Batch(descs, nrhs=2, rtol=1e-10, threads=512, ctas_per_sm=1,
                 bc=mb.SP_BC_PERIODIC if periodic else mb.SP_BC_AFFINE)
    for i, et in enumerate(ets):
        b.set_etype(i, et)
    stress, _, info = b.homogenize(np.ascontiguousarray(eps * strain))
    inf = mb.info_array(info)
    assert (inf["status"] == 0).all() and (inf["relres"] <= 1e-10).all(), inf
    for i, ref in enumerate(refs):
        assert np.abs(stress[i] - ref).max() <= 1e-8 * np.abs(ref).max(), meshes[i]


@pytest.mark.parametrize("k", [0, 2])
def test_breakdown_is_reported(k):
    """A strain whose forces leave FP32's range breaks its load case down: the
    RVE reports the residual that is not a number, whichever load case has it;
    the other RVE is solved."""
    descs = [mb.rve_desc(5, 0.3, (1e9, 2e10)), mb.rve_desc(4, 0.3, (1e9, 2e10))]
    eps = np.random.default_rng(2).normal(0, 1e-3, (2, 3, 6))
    eps[0, k] *= 1e38
    b = mb.Batch(descs, nrhs=3, threads=512, ctas_per_sm=1)
    b.upload(np.ascontiguousarray(eps))
    b.launch()
    info = (mb.sp_solve_info * 2)()
    b.download(np.zeros((2, 3, 6)), None, info)
    import torch
    torch.cuda.synchronize()
    assert info[0].status == mb.SP_ERR_NOCONV and np.isnan(info[0].relres)
    assert info[1].status == 0 and info[1].relres <= 1e-8
    b.close()


@pytest.mark.parametrize("cube", [True, False])
def test_periodic_fp64_edges(cube):
    """FP64 under periodic conditions: odd and even planes, rows across warps,
    the wide class, p and q or p alone on chip, and the first meshes past the
    range, on random voxel materials.  The periodic oracle's direct solve, and for
    the largest meshes the block stencil's FP64 batch; solves to 1e-10."""
    from oracle import periodic as PER
    rng = np.random.default_rng(53 + cube)
    meshes = PER_MESHES + [(18, 17, 13), (20, 20, 16), (18, 18, 30), (20, 20, 20), (24, 20, 22)]
    descs, ets, lens = [], [], []
    for n in meshes:
        edge = rng.uniform(0.05, 0.2, 3)
        lens.append([n[k] / 8.0 if cube else n[k] * edge[k] for k in range(3)])
        descs.append(mb.rve_desc(n, 0.2, (1e9, 1e9 * float(rng.uniform(2, 100))), (0.3, 0.25),
                                 lens[-1]))
        ets.append((rng.random(n[0] * n[1] * n[2]) < 0.4).astype(np.uint8))
    eps = rng.normal(0, 1e-3, (len(descs), 2, 6))
    out = []
    for ctas in (1, 2):
        b = mb.Batch(descs, nrhs=2, rtol=1e-10, bc=mb.SP_BC_PERIODIC, precision=mb.SP_PREC_FP64,
                     threads=512, ctas_per_sm=ctas)
        for i, et in enumerate(ets):
            b.set_etype(i, et)
        s, strain, info = b.homogenize(np.ascontiguousarray(eps))
        inf = mb.info_array(info)
        assert (inf["status"] == 0).all() and (inf["relres"] <= 1e-10).all()
        assert np.allclose(strain, eps, rtol=0, atol=1e-14)
        assert (b.last_launches() > 2) == (ctas == 1)
        out.append(s)
        b.close()
    for i, n in enumerate(meshes):
        ref = out[1][i]
        if np.prod(n) <= 1500:
            m = O.mesh(3, [v + 1 for v in n], lens[i])
            ref = PER.homogenize_periodic(m, ets[i], tuple(descs[i].E), tuple(descs[i].nu), eps[i])[1]
        assert np.abs(out[0][i] - ref).max() <= 1e-8 * np.abs(ref).max(), (n, cube)
