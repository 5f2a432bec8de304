"""The FP32 descriptor on blocked tables (csrc/desc_blk.cu) and on k-planar
tables (csrc/fused.cu) against the FP64 k-planar kernels on the same inputs:
one warp or four warps an atom (the lines lie at 8, 10 and, for the neighbours
in flight, 4 atoms for each of 152 SMs), full and partial 32-output blocks, an
odd and an even number of 16-output steps, short lists, and the layout of the
table copy.

Each FP32 quantity is a sum of at most a few hundred products with relative
errors of a few 2^-24 each: X, D and the forces agree with the FP64 kernels on
the same (FP32-valued) inputs within 2e-5 of the largest magnitude, the virial
(9 sums over all pairs) within 2e-5 of its largest component times the
cancellation in it (sum of magnitudes over magnitude, bounded by 10)."""

import importlib

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

_BUILT = {}


@pytest.fixture(scope="module")
def mods(gb):
    gb.load_library()
    return [importlib.import_module("dpmd_public_gb300." + m) for m in ("se_a", "model", "water")]


def _models(mods, width, sel):
    key = (width, sel)
    if key not in _BUILT:
        se_a, mdl, water = mods
        cfg = mdl.SeAConfig(neuron=(width // 4, width // 2, width), sel=sel, fitting=(32, 32))
        m64 = se_a.build_model(cfg, 5, [water.water_frame(4, 12.42, 700 + k) for k in range(2)],
                               DEV, torch.float64)
        m32 = se_a.SeAModel(cfg, m64.params_np, m64.davg.cpu().numpy(), m64.dstd.cpu().numpy(), DEV,
                            torch.float32, m64.tables_np, m64.infos_np)
        _BUILT[key] = m64, m32
    return _BUILT[key]


@pytest.mark.parametrize("mols", [1, 8, 202, 203, 405, 406, 506, 507])
@pytest.mark.parametrize("width,sel", [(100, (46, 92))])
def test_sizes(gb, mods, mols, width, sel):
    _check(gb, mods, mols, width, sel)


@pytest.mark.parametrize("mols", [64, 512])
@pytest.mark.parametrize("width,sel", [(16, (46, 92)), (20, (5, 7)), (32, (33, 1)), (36, (46, 92)),
                                       (48, (64, 31)), (64, (46, 92)), (68, (30, 60)),
                                       (96, (46, 92)), (112, (46, 92)), (128, (20, 200))])
def test_widths(gb, mods, mols, width, sel):
    _check(gb, mods, mols, width, sel)


@pytest.mark.parametrize("width,sel", [(16, (46, 92)), (20, (5, 7)), (36, (46, 92)), (128, (46, 92))])
def test_widths_between(gb, mods, width, sel):
    """900 atoms: four warps an atom in both directions (fewer take eight in
    the forward, more a warp an atom)."""
    _check(gb, mods, 300, width, sel)


def _descriptor(gb, m, dtype, form, b, em, dD, X=None):
    """X, D (X is None) or force, virial of one kernel form."""
    import ctypes

    L = gb._lib
    lib, cfg = L.load(), m.cfg
    P = lambda t: ctypes.c_void_p(t.data_ptr())
    M = cfg.neuron[-1]
    tabs = [m._blocked(t) if form == "blk" else m._planar(t) for t in m.tables]
    ptrs = (ctypes.c_void_p * len(tabs))(*[t.data_ptr() for t in tabs])
    head = (ptrs, m._tab_infos, cfg.ntypes, m._sel_c, int(cfg.type_one_side))
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    if X is None:
        X = torch.empty(b.nloc, 4, M, dtype=dtype, device=DEV)
        D = torch.empty(b.nloc, M * 16, dtype=dtype, device=DEV)
        tail = head + (b.nloc, M, 16, st)
        if form == "blk":
            rc = lib.gbdp_se_a_descriptor_fwd_blk_f32(P(X), P(D), None, None, P(em), P(b.atype),
                                                      None, *tail)
        else:
            rc = getattr(lib, "gbdp_se_a_descriptor_fwd_" + form)(P(X), P(D), P(em), P(b.atype),
                                                                  None, *tail)
        L.check(rc, "fwd")
        torch.cuda.synchronize()
        return X, D
    F = torch.empty(b.nloc, 3, dtype=dtype, device=DEV)
    V = torch.empty(b.nframes, 9, dtype=torch.float64, device=DEV)
    xc, isd = b.env.ext_coord.to(dtype), m.dstd_inv
    fn = lib.gbdp_se_a_descriptor_bwd_blk_f32 if form == "blk" else \
        getattr(lib, "gbdp_se_a_descriptor_bwd_" + form)
    L.check(fn(P(F), P(V), P(X), P(dD), None, P(em), P(b.env.nlist_ext), P(xc), P(b.env.ext_map),
               P(b.atype), P(isd), P(b.atom_frame), P(b.frame_aoff), P(b.frame_eoff), *head,
               ctypes.c_float(cfg.rcut_smth), ctypes.c_float(cfg.rcut), b.nloc, b.nframes, M, 16,
               None, st), "bwd")
    torch.cuda.synchronize()
    return F, V


def _check(gb, mods, mols, width, sel):
    se_a, mdl, water = mods
    m64, m32 = _models(mods, width, sel)
    side = int(np.ceil(mols ** (1 / 3) - 1e-9))
    box = float(np.float32(water.water_box_for(max(mols, 8))))
    c, t, _ = water.water_frame(side, box, 40 + mols, n_mol=mols)
    b = m32.batch([t], np.diag([box] * 3).reshape(1, 9))
    m32.step_fused(b, torch.tensor(c.astype(np.float32), device=DEV))  # fills the env rows
    assert b.status() == 0
    em = b.env.em
    X, D = _descriptor(gb, m64, torch.float64, "f64", b, em.double(), None)
    dD = (torch.randn(D.shape, generator=torch.Generator(device=DEV).manual_seed(mols), device=DEV)
          * 0.1)
    F, V = _descriptor(gb, m64, torch.float64, "f64", b, em.double(), dD.double(),
                       X.float().double())
    for form in ("blk", "f32"):
        x, d = _descriptor(gb, m32, torch.float32, form, b, em, None)
        f, v = _descriptor(gb, m32, torch.float32, form, b, em, dD, X.float())
        for name, got, ref, tol in (("X", x, X, 2e-5), ("D", d, D, 2e-5), ("F", f, F, 2e-5),
                                    ("V", v, V, 2e-4)):
            err = float((got.double() - ref).abs().max())
            assert err <= tol * float(ref.abs().max()), (form, name, err)


@pytest.mark.parametrize("mols", [13, 202, 203, 405, 406, 506, 507, 666])
@pytest.mark.parametrize("width,sel", [(100, (46, 92)), (48, (64, 31))])
def test_launch_shapes(gb, mods, mols, width, sel):
    """Every shape the tuner may keep, not only the untuned one, on both sides
    of the sharing lines (608, 1,520; backward 1,216 atoms): the bounds of the
    module, and D's FP16 parts against the FP32 form's D (a row's parts hold
    22 bits under a scale bounded by |X_k| |X_a|, 2^-21 of it)."""
    L = gb._lib
    lib = L.load()
    m64, m32 = _models(mods, width, sel)
    b, em = _env_rows(mods, m32, mols)
    X, D = _descriptor(gb, m64, torch.float64, "f64", b, em.double(), None)
    dD = torch.randn(D.shape, generator=torch.Generator(device=DEV).manual_seed(mols), device=DEV)
    F, V = _descriptor(gb, m64, torch.float64, "f64", b, em.double(), dD.double(),
                       X.float().double())
    key = (0, width, sum(sel), b.nloc)
    near = lambda got, ref, tol: float((got.double() - ref).abs().max()) <= tol * float(ref.abs().max())
    try:
        for warps in (1, 2, 4):
            L.check(lib.gbdp_autotune_set(0, 1, *key, warps, 1), "autotune_set")
            x, d = _descriptor(gb, m32, torch.float32, "blk", b, em, None)
            assert near(x, X, 2e-5) and near(d, D, 2e-5), warps
            xs, hi, lo, rs = _split_fwd(gb, m32, b, em)
            assert torch.equal(xs, x), warps
            nk = x.double().square().sum(1)
            bound = (nk.amax(1) * nk[:, :16].amax(1)).sqrt()[:, None]
            got = (hi.double() + lo.double()) * rs.double()[:, None]
            assert bool(((got - d.double()).abs() <= 2.0 ** -21 * bound).all()), warps
            for nbrs in (1, 2):
                L.check(lib.gbdp_autotune_set(1, 1, *key, warps, nbrs), "autotune_set")
                f, v = _descriptor(gb, m32, torch.float32, "blk", b, em, dD, X.float())
                assert near(f, F, 2e-5) and near(v, V, 2e-4), (warps, nbrs)
    finally:
        for bwd in (0, 1):
            L.check(lib.gbdp_autotune_set(bwd, 1, *key, 0, 1), "autotune_set")


def _split_fwd(gb, m, b, em):
    """X and D's FP16 parts with the rows' inverse scales."""
    import ctypes

    L = gb._lib
    cfg = m.cfg
    P = lambda t: ctypes.c_void_p(t.data_ptr())
    M = cfg.neuron[-1]
    tabs = [m._blocked(t) for t in m.tables]
    ptrs = (ctypes.c_void_p * len(tabs))(*[t.data_ptr() for t in tabs])
    X = torch.empty(b.nloc, 4, M, device=DEV)
    hi, lo = (torch.empty(b.nloc, M * 16, dtype=torch.float16, device=DEV) for _ in range(2))
    rs = torch.empty(b.nloc, device=DEV)
    L.check(L.load().gbdp_se_a_descriptor_fwd_blk_f32(
        P(X), P(hi), P(lo), P(rs), P(em), P(b.atype), None, ptrs, m._tab_infos, cfg.ntypes, m._sel_c,
        int(cfg.type_one_side), b.nloc, M, 16,
        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)), "fwd")
    torch.cuda.synchronize()
    return X, hi, lo, rs


def _env_rows(mods, m32, mols):
    """A batch of one frame of mols molecules and its env rows."""
    water = mods[2]
    side = int(np.ceil(mols ** (1 / 3) - 1e-9))
    box = float(np.float32(water.water_box_for(max(mols, 8))))
    c, t, _ = water.water_frame(side, box, 40 + mols, n_mol=mols)
    b = m32.batch([t], np.diag([box] * 3).reshape(1, 9))
    m32.step_fused(b, torch.tensor(c.astype(np.float32), device=DEV))
    assert b.status() == 0
    return b, b.env.em


@pytest.mark.parametrize("m", [100, 37, 16, 128])
def test_table_to_blocked_layout(gb, m):
    L = gb._lib
    lib = L.load()
    nrow = 5
    src_np = np.random.default_rng(3).standard_normal((nrow, 6 * m)).astype(np.float32)
    src = torch.tensor(src_np, device=DEV)
    re = lib.gbdp_table_blocked_row_elems(m)
    nb = (m + 31) // 32
    assert re == 192 * nb
    dst = torch.full((nrow * re,), 7.0, device=DEV)
    L.check(lib.gbdp_table_to_blocked_f32(dst.data_ptr(), src.data_ptr(), nrow, m, None),
            "table_to_blocked")
    torch.cuda.synchronize()
    co = np.zeros((nrow, 32 * nb, 6), np.float32)
    co[:, :m] = src_np.reshape(nrow, m, 6)
    # [row, block, half, t, plane, low / high coefficient] -> [row, block, plane, t, low / high, half]
    exp = co.reshape(nrow, nb, 2, 16, 3, 2).transpose(0, 1, 4, 3, 5, 2)
    np.testing.assert_array_equal(dst.cpu().numpy().reshape(exp.shape), exp)
