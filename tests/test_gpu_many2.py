"""Many steps per launch on small 2D grids (sp_many2.cuh) and the warp-strip 2D
step (sp_strip2.cuh): every step count and shape gives the bits of the one-step
tile kernel, on ragged and tiny grids, with periodic, constant and mixed sides
(different constants on each), batches, both dtypes and forms, all models, and
for ensembles of mixed members; the many-step kernel at chosen tiles and depths
(tiles that do not divide the grid, depths past the grid's own extent), the
state before the last step for moving windows' rims, and mass conservation."""
import numpy as np
import pytest

import symphas_b200 as sp

pytestmark = pytest.mark.gpu

P, D = sp.BoundaryType.PERIODIC, sp.BoundaryType.DEFAULT
MODELS = {"A": sp.model_MA_t, "B": sp.model_MB_t, "C": sp.model_MC_t, "AMK": sp.model_MAMK_t,
          "BMK": sp.model_MBMK_t}
WALLS = {"": [P] * 6, "x": [D, D, P, P, P, P], "y": [P, P, D, D, P, P], "xy": [D, D, D, D, P, P]}


def run(monkeypatch, env, model, dims, dtype, form, steps, walls="", batch=1, wide=False, chunks=(),
        conserve=0):
    for k in ("SP_TILE", "SP_MANY"):
        monkeypatch.delenv(k, raising=False)
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    st = sp.Stencil2d2h() if wide else sp.Stencil2d2h(5, 6, 13)
    params = sp.ProblemParameters(dims, boundary=WALLS[walls],
                                  boundary_value=[0.3, -0.2, 0.15, 0.05, 0.0, 0.0])
    m = MODELS[model](2, sp.SolverFT(st, form=form), params, coeff=(0.8, 1.1), dtype=dtype,
                      batch=batch)
    for i in range(batch):
        for f in range(m.nfields):
            m.fill_uniform(f, 31 + 7 * i + f, -0.3, 0.2, inst=i)
    if conserve:
        m.conserve_mass(conserve)
    for s in chunks or (steps,):
        m.step(0.01, s)
    out = np.stack([m.get_field(f, inst=i) for i in range(batch) for f in range(m.nfields)])
    info, launches = m.kernel_info(), m.launch_count()
    m.close()
    return out, info, launches


@pytest.mark.parametrize("model,dtype,form", [("A", "f64", "exact"), ("B", "f32", "fused"),
                                              ("B", "f64", "exact"), ("C", "f32", "fused"),
                                              ("C", "f64", "exact"), ("AMK", "f32", "fused"),
                                              ("BMK", "f64", "fused")])
@pytest.mark.parametrize("dims,many", [((64, 64), "16,8,8"), ((37, 21), "12,5,4"),
                                       ((9, 130), "8,40,3"), ((101, 53), "40,16,6")])
@pytest.mark.parametrize("walls", ["", "x", "y", "xy"])
def test_many_steps_match_single_steps(model, dtype, form, dims, many, walls, monkeypatch):
    want, info, n1 = run(monkeypatch, {"SP_MANY": "0"}, model, dims, dtype, form, 19, walls)
    assert info["steps_per_launch"] == 1 and n1 == 19
    got, info, n = run(monkeypatch, {"SP_MANY": many}, model, dims, dtype, form, 19, walls)
    assert info["steps_per_launch"] == int(many.split(",")[2]) and n < n1
    assert np.array_equal(got, want)


@pytest.mark.parametrize("dims,kw", [((64, 64), {}), ((16, 12), {}), ((300, 200), {"batch": 3}),
                                     ((255, 129), {"wide": True}), ((804, 601), {}),
                                     ((48, 48), {"conserve": 7}), ((70, 50), {"walls": "xy"})])
@pytest.mark.parametrize("model,dtype,form", [("A", "f32", "fused"), ("B", "f32", "fused"),
                                              ("B", "f64", "exact")])
def test_chosen_depth_matches_single_steps(model, dtype, form, dims, kw, monkeypatch):
    """The depth the library chooses, over calls of different lengths (graph
    replay, remainders, single steps)."""
    chunks = (1, 2, 600, 33, 5)
    want, _, _ = run(monkeypatch, {"SP_MANY": "0"}, model, dims, dtype, form, 0, chunks=chunks, **kw)
    got, info, _ = run(monkeypatch, {}, model, dims, dtype, form, 0, chunks=chunks, **kw)
    if dims == (64, 64):
        assert info["steps_per_launch"] > 1
    if kw.get("wide") and form == "fused":
        # the term order of the exact form compiled with contraction: which
        # products fuse is the compiler's choice per kernel, one rounding each
        assert np.abs(got - want).max() <= 641 * 2.0 ** -24
    else:
        assert np.array_equal(got, want)


def strip_variants(monkeypatch, model, dims):
    _, info, _ = run(monkeypatch, {"SP_TILE": "0"}, model, dims, "f32", "fused", 1)
    out = []
    for v in range(info["variants"]):
        _, i, _ = run(monkeypatch, {"SP_TILE": str(v)}, model, dims, "f32", "fused", 1)
        if i["variant"] == v and i["tile_x"] == 120:
            out.append(v)
    return out


@pytest.mark.parametrize("model", sorted(MODELS))
@pytest.mark.parametrize("dims", [(8, 9), (120, 40), (124, 33), (256, 64), (480, 17), (1000, 70)])
@pytest.mark.parametrize("walls", ["", "x", "xy"])
def test_strip_step_matches_tile_step(model, dims, walls, monkeypatch):
    vs = strip_variants(monkeypatch, model, (128, 64))
    assert vs
    want, _, _ = run(monkeypatch, {"SP_TILE": "0"}, model, dims, "f32", "fused", 9, walls, batch=2)
    for v in vs:
        got, info, _ = run(monkeypatch, {"SP_TILE": str(v)}, model, dims, "f32", "fused", 9, walls,
                           batch=2)
        assert info["variant"] == v
        assert np.array_equal(got, want)
    # ragged rows, and rows a group of which lies at both faces, keep the tile kernel
    for d in ((130, 40), (4, 40)):
        _, info, _ = run(monkeypatch, {"SP_TILE": str(vs[0])}, model, d, "f32", "fused", 1)
        assert info["variant"] == 0


def test_strip_step_on_ensembles(monkeypatch):
    members = sp.ensemble_members(12, seed=3, sides=(64, 96, 128, 256, 384))
    outs = {}
    e = sp.Ensemble(sp.SolverFT(sp.Stencil2d2h(5, 6, 13)), members)
    nv = e.kernel_info()["variants"]
    e.close()
    for v in range(nv):
        monkeypatch.setenv("SP_TILE", str(v))
        e = sp.Ensemble(sp.SolverFT(sp.Stencil2d2h(5, 6, 13)), members)
        if e.kernel_info()["variant"] == v and (v == 0 or e.kernel_info()["tile_x"] == 120):
            for i in range(len(members)):
                e.fill_uniform(0, 5 + i, -0.1, 0.1, inst=i)
            e.step(41)
            outs[v] = [e.get_field(0, inst=i) for i in range(len(members))]
        e.close()
    assert len(outs) > 1
    for v in outs:
        for a, b in zip(outs[0], outs[v]):
            assert np.array_equal(a, b), v


@pytest.mark.parametrize("dim,dims", [(2, (64, 48)), (2, (300, 200)), (3, (20, 16, 12))])
@pytest.mark.parametrize("model,dtype,form", [("A", "f32", "fused"), ("C", "f64", "exact")])
def test_constant_sides_before_the_first_upload(dim, dims, model, dtype, form):
    """Steps from a handle's zero state: the same fields whether the steps come
    in one call or one by one, and as after an upload of zeros."""
    st = sp.Stencil2d2h(5, 6, 13) if dim == 2 else sp.Stencil3d2h(7, 10, 25)
    params = sp.ProblemParameters(dims, boundary=WALLS["xy"],
                                  boundary_value=[0.3, -0.2, 0.15, 0.05, 0.0, 0.0])
    outs = []
    for upload, chunks in ((True, (1,) * 6), (False, (1,) * 6), (False, (6,))):
        m = MODELS[model](dim, sp.SolverFT(st, form=form), params, coeff=(0.8, 1.1), dtype=dtype,
                          batch=2)
        if upload:
            for i in range(2):
                for f in range(m.nfields):
                    m.set_field(f, np.zeros(dims[::-1]), inst=i)
        for s in chunks:
            m.step(0.002, s)
        outs.append(np.stack([m.get_field(f, inst=i) for i in range(2) for f in range(m.nfields)]))
        m.close()
    assert np.abs(outs[0]).max() > 0
    assert np.array_equal(outs[0], outs[1]) and np.array_equal(outs[0], outs[2])


@pytest.mark.parametrize("model,dims", [("A", (256, 256)), ("B", (804, 601)), ("B", (1024, 512)),
                                        ("C", (640, 480)), ("A", (1024, 1024))])
def test_later_handles_start_as_the_tuner_left_one(model, dims, monkeypatch):
    """The tuner's answer about the many-step kernel, and not the estimate that
    it may have overruled, is what later handles of the same grid start with."""
    for k in ("SP_TILE", "SP_MANY"):
        monkeypatch.delenv(k, raising=False)
    got = []
    for tune in (True, False):
        m = MODELS[model](2, sp.SolverFT(sp.Stencil2d2h(5, 6, 13), form="fused"),
                          sp.ProblemParameters(dims, boundary=[P] * 6), dtype="f32")
        if tune:
            m.autotune(5)
        i = m.kernel_info()
        got.append((i["variant"], i["steps_per_launch"]))
        m.close()
    assert got[0] == got[1]


@pytest.mark.parametrize("model", sorted(MODELS))
@pytest.mark.parametrize("dtype,form,wide", [("f32", "fused", True), ("f64", "fused", True),
                                             ("f32", "exact", True), ("f32", "exact", False),
                                             ("f64", "exact", True), ("f32", "fused", False)])
@pytest.mark.parametrize("dims,walls", [((64, 64), ""), ((101, 53), "x"), ((300, 200), "")])
def test_bits_do_not_depend_on_the_calls(model, dtype, form, wide, dims, walls, monkeypatch):
    """A run in one call, in single steps and in uneven calls: the same bits, on
    every point set of the dispatch."""
    if wide and form == "fused" and model in ("AMK", "BMK"):
        pytest.skip("no such kernel")
    outs = [run(monkeypatch, {}, model, dims, dtype, form, 0, walls, wide=wide, chunks=c)[0]
            for c in ((25,), (1,) * 25, (7, 1, 13, 4))]
    assert np.array_equal(outs[0], outs[1]) and np.array_equal(outs[0], outs[2])
