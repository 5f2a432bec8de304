"""BF16 tensor-core embedding of the uncompressed se_e2_a descriptor
(csrc/embed_tc.cu) against the FP32 torch embedding of the same model, and
the whole tensor-core plain step against the FP64 CPU composite.

Stated tolerances (BF16 MMA operands with FP32 accumulation, tanh.approx;
relative to the largest magnitude of the reference):
  X and D:            max |diff| <= 1e-2 max |ref|
  dE/d(env matrix):   max |diff| <= 2e-2 max |ref|
  plain-tc step vs FP64: |dF| <= 2e-2 eV/A, |dE| / natoms <= 1e-3 eV
The measured errors are printed."""

import importlib

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def setup(gb):
    gb.load_library()
    se_a = importlib.import_module("dpmd_public_gb300.se_a")
    mdl = importlib.import_module("dpmd_public_gb300.model")
    water = importlib.import_module("dpmd_public_gb300.water")
    cfg = mdl.SeAConfig()
    stat = [water.water_frame(4, 12.42, 1000 + s) for s in range(4)]
    m64 = se_a.build_model(cfg, 7, stat, DEV, torch.float64)
    args = (cfg, m64.params_np, m64.davg.cpu().numpy(), m64.dstd.cpu().numpy(), DEV, torch.float32)
    return se_a, water, cfg, m64, se_a.SeAModel(*args), se_a.SeAModel(*args, fit_mode="tc-f16x3")


def _ref_x(model, em, atype):
    """X [n, 4, M] of the FP32 torch embedding (the plain form's nets)."""
    cfg = model.cfg
    n, sec, M = em.shape[0], cfg.sec, cfg.neuron[-1]
    X = torch.zeros((n, 4, M), dtype=em.dtype, device=em.device)
    for tj in range(cfg.ntypes):
        for ti in ([None] if cfg.type_one_side else range(cfg.ntypes)):
            k = tj if cfg.type_one_side else tj * cfg.ntypes + ti
            rows = torch.arange(n, device=em.device) if ti is None else torch.nonzero(atype == ti)[:, 0]
            rr = em[rows, sec[tj]:sec[tj + 1], :]
            g = rr[:, :, :1]
            for w, b, skip in model.emb[k]:
                y = torch.tanh(g @ w + b)
                if skip == "same":
                    y = y + g
                elif skip == "double":
                    y = y + torch.cat([g, g], -1)
                g = y
            X = X.index_add(0, rows, rr.transpose(1, 2) @ g)
    return X / cfg.nnei


def _case(setup, mdl_idx, seed=5, n=4, L=12.42):
    se_a, water, cfg, m64, m32, m32tc = setup
    m = (m32, m32tc)[mdl_idx]
    c, t, b = water.water_frame(n, L, seed)
    batch = m.batch([t], b[None])
    coord = torch.tensor(c, dtype=torch.float32, device=DEV)
    batch.ensure_plain_tc(m)
    env = se_a.env_mat_packed(batch.plan, coord, batch.atype, m.davg, m.dstd, cfg.rcut_smth,
                              list(cfg.sel), out=batch.env_full)
    return m, batch, env, (c, t, b)


@pytest.mark.parametrize("mdl_idx", [0, 1])
def test_forward_x_and_d(setup, mdl_idx):
    m, batch, env, _ = _case(setup, mdl_idx)
    cfg = m.cfg
    m.embed_tc_forward(batch, env.em)
    torch.cuda.synchronize()
    assert int(batch.emb_status.item()) == 0
    Xr = _ref_x(m, env.em, batch.atype)
    ex = float((batch.X - Xr).abs().max() / Xr.abs().max())
    A = cfg.axis_neuron
    Dr = torch.einsum("ncm,nca->nma", Xr, Xr[:, :, :A]).reshape(batch.nloc, -1)
    D = batch.descriptor_rows()[batch.drow.long()]
    ed = float((D - Dr).abs().max() / Dr.abs().max())
    print(f"X rel err {ex:.3e}, D rel err {ed:.3e}")
    assert ex <= 1e-2 and ed <= 1e-2


def test_backward_env_gradient(setup):
    m, batch, env, _ = _case(setup, 0, seed=8)
    cfg = m.cfg
    m.embed_tc_forward(batch, env.em)
    gen = torch.Generator(device=DEV).manual_seed(2)
    batch.dD.copy_(torch.randn(batch.dD.shape, generator=gen, device=DEV))
    net = m.embed_tc_backward(batch, env.em)
    torch.cuda.synchronize()
    assert int(batch.emb_status.item()) == 0
    em = env.em.clone().requires_grad_(True)
    Xr = _ref_x(m, em, batch.atype)
    A = cfg.axis_neuron
    Dr = torch.einsum("ncm,nca->nma", Xr, Xr[:, :, :A]).reshape(batch.nloc, -1)
    g = torch.autograd.grad(Dr, em, grad_outputs=batch.dD[batch.drow.long()])[0]
    e = float((net - g).abs().max() / g.abs().max())
    print(f"dE/d(env) rel err {e:.3e}")
    assert e <= 2e-2


@pytest.mark.parametrize("mdl_idx", [0, 1])
def test_plain_tc_step_vs_fp64(setup, mdl_idx):
    import composite

    se_a, water, cfg, m64, m32, m32tc = setup
    m, batch, env, (c, t, b) = _case(setup, mdl_idx, seed=11)
    E, F, V = m.step_plain_tc(batch, torch.tensor(c, dtype=torch.float32, device=DEV))
    torch.cuda.synchronize()
    assert int(batch.emb_status.item()) == 0
    Er, Fr, Vr, _ = composite.energy_force_virial(cfg, m64.params_np, m64.davg.cpu().numpy(),
                                                  m64.dstd.cpu().numpy(), c, t, b, None, None)
    ef = float(np.abs(F.cpu().numpy().astype(np.float64) - Fr).max())
    ee = abs(float(E[0]) - Er) / len(t)
    ev = float(np.abs(V[0].cpu().numpy() - Vr).max())
    print(f"plain-tc vs FP64: |dF| {ef:.3e} eV/A (max |F| {np.abs(Fr).max():.3f}), "
          f"|dE|/N {ee:.3e} eV, |dV| {ev:.3e} eV")
    assert ef <= 2e-2 and ee <= 1e-3


@pytest.mark.parametrize("one_side,mols", [(True, 1), (True, 5), (False, 5), (False, 12)])
def test_equal_rows_and_slabs(setup, one_side, mols):
    """Sections whose equal rows at the end start at every edge of the 32-row
    slabs (none, all, one row off either side), odd numbers of atoms of a
    type (units without a second atom), nets per type and per type pair:
    X and dE/d(env matrix) against the FP32 torch embedding, with the
    tolerances stated above (BF16 operands)."""
    se_a, water, cfg0, m64, _, _ = setup
    import dataclasses

    cfg = dataclasses.replace(cfg0, type_one_side=one_side)
    mdl = importlib.import_module("dpmd_public_gb300.model")
    m = se_a.SeAModel(cfg, mdl.init_params(cfg, 3), m64.davg.cpu().numpy(),
                      m64.dstd.cpu().numpy(), DEV, torch.float32)
    atype = np.tile(np.array([0, 1, 1], np.int32), mols)
    b = m.batch([atype], np.diag([30.0] * 3).reshape(1, 9))
    b.ensure_plain_tc(m)
    g = torch.Generator(device=DEV).manual_seed(mols)
    em = torch.randn(b.nloc, cfg.nnei, 4, generator=g, device=DEV)
    edges = {46: [1, 2, 31, 32, 33, 34, 45, 46], 92: [1, 32, 33, 64, 65, 66, 91, 92]}
    for i in range(b.nloc):
        for t in range(2):
            k = edges[cfg.sel[t]][(i + 3 * t) % 8]  # rows k - 1 .. are equal
            em[i, cfg.sec[t] + k:cfg.sec[t + 1]] = torch.tensor([-0.4, 0.0, 0.0, 0.0], device=DEV)
            em[i, cfg.sec[t] + k - 1] = em[i, cfg.sec[t + 1] - 1] if k < cfg.sel[t] else em[i, 0]
    b.dD.copy_(torch.randn(b.dD.shape, generator=g, device=DEV) * 0.05)
    m.embed_tc_forward(b, em)
    net = m.embed_tc_backward(b, em)
    torch.cuda.synchronize()
    assert int(b.emb_status.item()) == 0
    x = em.clone().requires_grad_(True)
    Xr = _ref_x(m, x, b.atype)
    assert float((b.X - Xr).abs().max()) <= 1e-2 * float(Xr.abs().max())
    Dr = torch.einsum("ncm,nca->nma", Xr, Xr[:, :, :cfg.axis_neuron]).reshape(b.nloc, -1)
    ref = torch.autograd.grad(Dr, x, b.dD[b.drow.long()])[0]
    assert float((net - ref).abs().max()) <= 2e-2 * float(ref.abs().max())


@pytest.mark.parametrize("one_side", [True, False])
def test_one_and_two_units_a_block_agree(setup, one_side):
    """Few units take a block each, an atom's slabs on two warps; many, two
    a block: the same bits, X, D and dE/d(env matrix), for 41 molecules by
    themselves (62 units) and as the first of 210 (315)."""
    se_a, water, cfg0, m64, _, _ = setup
    import dataclasses

    cfg = dataclasses.replace(cfg0, type_one_side=one_side)
    mdl = importlib.import_module("dpmd_public_gb300.model")
    m = se_a.SeAModel(cfg, mdl.init_params(cfg, 3), m64.davg.cpu().numpy(),
                      m64.dstd.cpu().numpy(), DEV, torch.float32)
    g = torch.Generator(device=DEV).manual_seed(5)
    em = torch.randn(630, cfg.nnei, 4, generator=g, device=DEV)
    dD = torch.randn(630, cfg.neuron[-1] * cfg.axis_neuron, generator=g, device=DEV) * 0.05
    cut = torch.randint(1, 46, (630, 2), generator=g, device=DEV).tolist()
    for i, ks in enumerate(cut):  # equal rows from a random place on
        for t in range(2):
            em[i, cfg.sec[t] + ks[t] * (t + 1):cfg.sec[t + 1]] = torch.tensor([-0.4, 0., 0., 0.],
                                                                              device=DEV)
    got = []
    for mols in (41, 210):
        n = 3 * mols
        b = m.batch([np.tile(np.array([0, 1, 1], np.int32), mols)],
                    np.diag([60.0] * 3).reshape(1, 9))
        b.ensure_plain_tc(m)
        b.dD.zero_()
        b.dD[b.drow.long()] = dD[:n]
        e = em[:n].contiguous()
        m.embed_tc_forward(b, e)
        net = m.embed_tc_backward(b, e)
        torch.cuda.synchronize()
        assert int(b.emb_status.item()) == 0
        D = b.D[b.drow.long()]
        lo = getattr(b, "D_lo", None)
        parts = [b.X, net, D] + ([] if lo is None else [lo[b.drow.long()], b.D_rs[b.drow.long()]])
        got.append([q[:123].clone() for q in parts])
    for a, c in zip(*got):
        assert torch.equal(a, c)


@pytest.mark.parametrize("mols", [2, 210])
def test_nan_in_a_padding_row(setup, mols):
    """A row with s = NaN (0 / 0 in the statistics) makes every component of
    its atom's X NaN, its zero components too (0 NaN = NaN in the sum over the
    rows), also where the row is padding and evaluated for the equal rest; other
    atoms keep their bits."""
    se_a, water, cfg, m64, _, _ = setup
    mdl = importlib.import_module("dpmd_public_gb300.model")
    m = se_a.SeAModel(cfg, mdl.init_params(cfg, 3), m64.davg.cpu().numpy(),
                      m64.dstd.cpu().numpy(), DEV, torch.float32)
    n = 3 * mols
    b = m.batch([np.tile(np.array([0, 1, 1], np.int32), mols)], np.diag([60.0] * 3).reshape(1, 9))
    b.ensure_plain_tc(m)
    g = torch.Generator(device=DEV).manual_seed(2)
    em = torch.randn(n, cfg.nnei, 4, generator=g, device=DEV)
    for t in range(2):
        em[:, cfg.sec[t] + 20:cfg.sec[t + 1]] = torch.tensor([-0.4, 0., 0., 0.], device=DEV)
    m.embed_tc_forward(b, em)
    clean = b.X.clone()
    bad = torch.zeros(n, dtype=torch.bool, device=DEV)
    for i, t in ((0, 0), (4, 1), (n - 1, 0)):
        em[i, cfg.sec[t + 1] - 1, 0] = float("nan")
        bad[i] = True
    m.embed_tc_forward(b, em)
    torch.cuda.synchronize()
    assert int(b.emb_status.item()) == 0
    assert bool(torch.isnan(b.X[bad]).all())
    assert torch.equal(b.X[~bad], clean[~bad])
