"""End-to-end energy / force / virial of the three GPU forms against the FP64
CPU composite (oracle/composite.py, the reference's op sequence).

Stated tolerances (the FP32 bar is a force error <= 1e-5 eV/A vs FP64):
  fp64 GPU: |dF| <= 1e-9 eV/A, |dE| / natoms <= 1e-10 eV, |dV| <= 1e-8 eV
  fp32 GPU: |dF| <= 1e-5 eV/A, |dE| / natoms <= 1e-6 eV, |dV| <= 1e-3 eV
"""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def mods(gb):
    gb.load_library()
    import importlib

    return (importlib.import_module("dpmd_public_gb300.se_a"),
            importlib.import_module("dpmd_public_gb300.model"),
            importlib.import_module("dpmd_public_gb300.water"))


@pytest.fixture(scope="module")
def built(mods):
    se_a, mdl, water = mods
    cfg = mdl.SeAConfig()
    stat = [water.water_frame(4, 12.42, 1000 + s) for s in range(4)]
    m64 = se_a.build_model(cfg, 7, stat, DEV, torch.float64)
    m32 = se_a.SeAModel(cfg, m64.params_np, m64.davg.cpu().numpy(), m64.dstd.cpu().numpy(), DEV,
                        torch.float32, m64.tables_np, m64.infos_np)
    return cfg, m64, m32


TOL = {torch.float64: (1e-9, 1e-10, 1e-8), torch.float32: (1e-5, 1e-6, 1e-3)}


def _ref(composite, cfg, m, frame, compressed=True):
    c, t, b = frame
    return composite.energy_force_virial(cfg, m.params_np, m.davg.cpu().numpy(), m.dstd.cpu().numpy(),
                                         c, t, b, m.tables_np if compressed else None,
                                         m.infos_np if compressed else None)


def _check(E, F, V, ref, natoms, dtype):
    ft, et, vt = TOL[dtype]
    Er, Fr, Vr, _ = ref
    assert abs(float(E) - Er) / natoms <= et, (float(E), Er)
    assert np.abs(F - Fr).max() <= ft, np.abs(F - Fr).max()
    assert np.abs(V - Vr).max() <= vt, np.abs(V - Vr).max()


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("form", ["fused", "ops", "plain"])
def test_forms_vs_fp64_composite(mods, built, dtype, form):
    import composite

    se_a, mdl, water = mods
    cfg, m64, m32 = built
    m = m64 if dtype == torch.float64 else m32
    frame = water.water_frame(4, 12.42, 5)
    b = m.batch([frame[1]], frame[2][None])
    coord = torch.tensor(frame[0], dtype=dtype, device=DEV)
    if form == "fused":
        E, F, V = m.step_fused(b, coord)
        assert b.status() == 0
    else:
        E, F, V = m.step_ops(b, coord, compressed=(form == "ops"))
    ref = _ref(composite, cfg, m64, frame, compressed=(form != "plain"))
    _check(E[0].item(), F.detach().cpu().numpy().astype(np.float64), V[0].cpu().numpy(), ref,
           len(frame[1]), dtype)


def test_fused_ragged_batch(mods, built):
    import composite

    se_a, mdl, water = mods
    cfg, m64, m32 = built
    frames = water.ragged_frames(5, seed=11, lo=8, hi=120)
    b = m32.batch([f[1] for f in frames], np.stack([f[2] for f in frames]))
    coord = torch.tensor(np.concatenate([f[0] for f in frames]), dtype=torch.float32, device=DEV)
    E, F, V = m32.step_fused(b, coord)
    Fn = F.cpu().numpy().astype(np.float64)
    off = 0
    for k, fr in enumerate(frames):
        n = len(fr[1])
        _check(E[k].item(), Fn[off:off + n], V[k].cpu().numpy(), _ref(composite, cfg, m64, fr), n,
               torch.float32)
        off += n


def test_fused_graph_replay_matches_eager(mods, built):
    se_a, mdl, water = mods
    cfg, m64, m32 = built
    frame = water.water_frame(4, 12.42, 9)
    b = m32.batch([frame[1]], frame[2][None])
    coord = torch.tensor(frame[0], dtype=torch.float32, device=DEV)
    E0, F0, V0 = (x.clone() for x in m32.step_fused(b, coord))
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        for _ in range(2):
            m32.step_fused(b, coord)
    torch.cuda.current_stream().wait_stream(s)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        out = m32.step_fused(b, coord)
    coord.add_(0.0)
    g.replay()
    torch.cuda.synchronize()
    assert torch.allclose(out[0], E0, rtol=1e-6, atol=1e-6)
    assert torch.allclose(out[1], F0, rtol=1e-4, atol=1e-6)
    assert b.status() == 0


@pytest.mark.parametrize("mode,ftol", [("fp32", 1e-5), ("tf32x3", 1e-5), ("native-fp32", 1e-5),
                                       ("native-bf16x9", 1e-5), ("native-tf32", 5e-3),
                                       ("bf16", 5e-3), ("native-bf16", 5e-3)])
def test_fused_fitting_modes(mods, built, mode, ftol):
    """The fused form with each fitting GEMM mode vs the FP64 composite.
    FP32-level modes meet the 1e-5 eV/A force bar; TF32 / BF16 state 5e-3."""
    import composite

    se_a, mdl, water = mods
    cfg, m64, m32 = built
    m = se_a.SeAModel(cfg, m64.params_np, m64.davg.cpu().numpy(), m64.dstd.cpu().numpy(), DEV,
                      torch.float32, m64.tables_np, m64.infos_np, fit_mode=mode)
    frame = water.water_frame(4, 12.42, 5)
    b = m.batch([frame[1]], frame[2][None])
    E, F, V = m.step_fused(b, torch.tensor(frame[0], dtype=torch.float32, device=DEV))
    Er, Fr, Vr, _ = _ref(composite, cfg, m64, frame)
    err = np.abs(F.cpu().numpy().astype(np.float64) - Fr).max()
    assert err <= ftol, (mode, err)
    assert abs(float(E[0]) - Er) / len(frame[1]) <= (1e-6 if ftol <= 1e-5 else 1e-3)


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_forward_lower_matches_fused(mods, built, dtype):
    """The forward_lower path (extended coordinates + an unsorted rcut + skin
    list from an MD engine, formatted on the GPU, op-form descriptor and
    fitting, ghost forces folded through the mapping) gives the fused step's
    energy, forces and virial on the same frame."""
    import os

    se_a, mdl, water = mods
    cfg, m64, m32 = built
    m = m64 if dtype == torch.float64 else m32
    g = np.load(os.path.join(os.path.dirname(__file__), "golden", "pt_format_nlist.npz"))
    nloc = int(g["nloc"])
    T = lambda a, dt=dtype: torch.tensor(a, dtype=dt, device=DEV)
    El, Fl, Vl = m.step_lower(T(g["ext_coord"]), T(g["ext_type"], torch.int32),
                              T(g["nlist_in"], torch.int32), T(g["mapping"], torch.int64), nloc)
    b = m.batch([g["atype"]], g["box"][None])
    Ef, Ff, Vf = m.step_fused(b, T(g["coord"]))
    ft, et, vt = TOL[dtype]
    assert abs(float(El) - float(Ef[0])) / nloc <= et
    assert float((Fl - Ff).abs().max()) <= ft
    assert float((Vl - Vf[0]).abs().max()) <= vt


@pytest.mark.parametrize("dtype,compressed,tol", [(torch.float64, False, (1e-10, 1e-10, 1e-10)),
                                                   (torch.float32, False, (1e-5, 2e-5, 2e-5)),
                                                   (torch.float64, True, (1e-10, 1e-10, 1e-10)),
                                                   (torch.float32, True, (1e-5, 2e-5, 2e-5))])
def test_reference_model_testcase(mods, dtype, compressed, tol):
    """The reference's se_e2_a test model (deeppot_sea.yaml) through the
    operator form on the GPU reproduces its own inference test values
    (deeppot-testcase.yaml).  Stated tolerances (per-atom energy, force,
    virial): FP64 1e-10, plain and compressed (tables at the reference's
    default 0.01 / 0.1 strides: the FP64 CPU composite of the compressed model
    is within 1e-14 of these values); FP32 1e-5 / 2e-5 / 2e-5 (atomic
    energies near -93 and -186 eV carry FP32 rounding of ~1e-5)."""
    import importlib
    import os

    se_a, mdl, water = mods
    S = importlib.import_module("dpmd_public_gb300.serial")
    g = np.load(os.path.join(os.path.dirname(__file__), "golden", "ref_deeppot_sea.npz"))
    cfg, params, davg, dstd, _ = S.unflatten(dict(g))
    tables = infos = None
    if compressed:
        tables, infos = mdl.build_tables(params, davg, dstd, 0.9, cfg)
    m = se_a.SeAModel(cfg, params, davg, dstd, DEV, dtype, tables, infos)
    et, ft, vt = tol
    for n in range(int(g["ncases"])):
        c = g[f"case{n}_coord"].reshape(-1, 3)
        t = g[f"case{n}_atype"].astype(np.int32)
        b = g[f"case{n}_box"] if f"case{n}_box" in g.files else np.diag([100.0] * 3).reshape(-1)
        bt = m.batch([t], np.asarray(b).reshape(1, 9))
        E, F, V = m.step_ops(bt, torch.tensor(c, dtype=dtype, device=DEV), compressed=compressed)
        ae = g[f"case{n}_atomic_energy"]
        assert abs(float(E[0]) - ae.sum()) / len(t) <= et, (n, float(E[0]), ae.sum())
        assert np.abs(F.cpu().numpy() - g[f"case{n}_force"].reshape(-1, 3)).max() <= ft
        v_ref = g[f"case{n}_atomic_virial"].reshape(-1, 9).sum(0)
        assert np.abs(V[0].cpu().numpy() - v_ref).max() <= vt


def test_autotuned_launch_shape(mods, built):
    """Launch-shape autotuning of the fused descriptor kernels: the first
    uncaptured call of a new shape times 1, 2 and 4 centres per CTA (and for
    the backward 1 or 2 neighbours in flight per 16-lane group) and keeps the
    fastest; the step's results do not depend on the choice, and a CUDA
    graph captured afterwards uses the tuned shape."""
    L = __import__("dpmd_public_gb300._lib", fromlist=["x"])
    se_a, mdl, water = mods
    cfg, m64, m32 = built
    frame = water.water_frame(3, 9.315, 21)  # 81 atoms: a shape no other test uses
    b = m32.batch([frame[1]], frame[2][None])
    coord = torch.tensor(frame[0], dtype=torch.float32, device=DEV)
    E0, F0, V0 = (x.clone() for x in m32.step_fused(b, coord))
    L.set_autotune(True)
    try:
        E1, F1, V1 = (x.clone() for x in m32.step_fused(b, coord))
    finally:
        L.set_autotune(False)
    rep = L.autotune_report()
    mine = [l for l in rep if "nloc=2^6" in l and "f32 M=100 nnei=138" in l]
    assert {l.split()[0] for l in mine} == {"se_a_descriptor_fwd", "se_a_descriptor_bwd"}, rep
    for l in mine:
        assert int(l.split("warps=")[1].split()[0]) in (1, 2, 4)
        if l.startswith("se_a_descriptor_bwd"):  # neighbours in flight per 16-lane group
            assert int(l.split("nbrs=")[1].split()[0]) in (1, 2)
            assert len(l.split("ms=")[1].split(",")) == 6
    assert torch.allclose(E1, E0, rtol=1e-6, atol=1e-6)
    assert torch.allclose(F1, F0, rtol=1e-5, atol=1e-6)
    g = torch.cuda.CUDAGraph()
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        m32.step_fused(b, coord)
    torch.cuda.current_stream().wait_stream(s)
    with torch.cuda.graph(g):
        out = m32.step_fused(b, coord)
    g.replay()
    torch.cuda.synchronize()
    assert torch.allclose(out[1], F0, rtol=1e-5, atol=1e-6)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_fused_deterministic_mode(mods, built, dtype):
    """step_fused(deterministic=True): forces, virials and energies summed in
    64-bit fixed point are the same bits on every run (also across a CUDA
    graph replay), agree with the atomic sums within the FP32 / FP64
    rounding, and keep the stated tolerances against the FP64 composite."""
    import composite

    se_a, mdl, water = mods
    cfg, m64, m32 = built
    m = m64 if dtype == torch.float64 else m32
    frame = water.water_frame(4, 12.42, 13)
    b = m.batch([frame[1]], frame[2][None])
    coord = torch.tensor(frame[0], dtype=dtype, device=DEV)
    runs = [tuple(x.clone() for x in m.step_fused(b, coord, deterministic=True)) for _ in range(3)]
    for r in runs[1:]:
        for a, c in zip(r, runs[0]):
            assert torch.equal(a, c)
    Ea, Fa, Va = (x.clone() for x in m.step_fused(b, coord))
    E, F, V = runs[0]
    # fixed-point grid per term: 2^-40 eV/A (FP64), 2^-32 (FP32), ~100 terms per atom
    ft = 1e-10 if dtype == torch.float64 else 1e-6
    assert float((F - Fa).abs().max()) <= ft
    assert float((E - Ea).abs().max()) <= 1e-8
    assert float((V - Va).abs().max()) <= (1e-9 if dtype == torch.float64 else 1e-4)
    _check(E[0].item(), F.cpu().numpy().astype(np.float64), V[0].cpu().numpy(),
           _ref(composite, cfg, m64, frame), len(frame[1]), dtype)
    # a graph captured in this mode replays the same bits
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        m.step_fused(b, coord, deterministic=True)
    torch.cuda.current_stream().wait_stream(s)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        out = m.step_fused(b, coord, deterministic=True)
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(out[1], F) and torch.equal(out[0], E) and torch.equal(out[2], V)


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("det", [0, 1])
@pytest.mark.parametrize("nrows,nframes", [(1, 1), (33, 40), (2047, 3), (2048, 300), (2049, 3),
                                           (5000, 17)])
def test_frame_energies(mods, dtype, det, nrows, nframes):
    """Rows of frames in any order and padding rows (frame -1), at the row
    counts where one block takes over from a grid, over an output that held
    other values: sums within n u of the magnitudes' (u = 2^-53), plus the
    fixed point's half step a row (2^-31) in the deterministic mode."""
    import importlib

    L = importlib.import_module("dpmd_public_gb300._lib")
    lib = L.load()
    g = torch.Generator(device=DEV).manual_seed(nrows)
    ae = torch.randn(nrows, generator=g, device=DEV, dtype=dtype)
    f = torch.randint(-1, nframes, (nrows,), generator=g, device=DEV, dtype=torch.int32)
    E = torch.full((nframes,), 7.0, device=DEV, dtype=torch.float64)
    fn = lib.gbdp_frame_energy_f64 if dtype == torch.float64 else lib.gbdp_frame_energy_f32
    rc = fn(E.data_ptr(), ae.data_ptr(), f.data_ptr(), nrows, nframes, det,
            torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    ok = (f >= 0).double()
    z = torch.zeros(nframes, device=DEV, dtype=torch.float64)
    ref = z.clone().index_add_(0, f.clamp_min(0).long(), ae.double() * ok)
    mag = z.clone().index_add_(0, f.clamp_min(0).long(), ae.double().abs() * ok)
    bound = 2 * nrows * 2.0 ** -53 * mag + (nrows * 2.0 ** -31 if det else 0.0)
    assert bool(((E - ref).abs() <= bound).all())


@pytest.mark.parametrize("n", [4, 7, 8])
def test_tuned_shapes_give_the_same_bits(mods, built, n):
    """The launch shapes the tuner chooses between (1, 2 or 4 warps, 1 or 2
    neighbours in flight) give a deterministic step the same bits, where warps
    share an atom (192 and 1,029 atoms) and where each has its own (1,536): the
    tuner's choice is by time, so results that depended on it
    would not be the same on every run."""
    L = __import__("dpmd_public_gb300._lib", fromlist=["x"])
    se_a, mdl, water = mods
    cfg, m64, m32 = built
    lib = L.load()
    frame = water.water_frame(n, 3.105 * n, 40 + n)
    b = m32.batch([frame[1]], frame[2][None])
    coord = torch.tensor(frame[0], dtype=torch.float32, device=DEV)
    key = (0, cfg.neuron[-1], sum(cfg.sel), b.nloc)
    run = lambda: tuple(x.clone() for x in m32.step_fused(b, coord, deterministic=True))
    ref = run()
    try:
        for bwd, warps, nbrs in [(0, 1, 1), (0, 2, 1), (0, 4, 1)] + [
                (1, w, u) for w in (1, 2, 4) for u in (1, 2)]:
            L.check(lib.gbdp_autotune_set(bwd, 1, *key, warps, nbrs), "autotune_set")
            for x, y in zip(run(), ref):
                assert torch.equal(x, y), (bwd, warps, nbrs)
    finally:
        for bwd in (0, 1):
            L.check(lib.gbdp_autotune_set(bwd, 1, *key, 0, 1), "autotune_set")
