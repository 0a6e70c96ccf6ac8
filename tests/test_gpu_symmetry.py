"""Kernels of the symmetry-adapted path at the sizes where they can go wrong:
chunks cut by pieces of the polynomial, the one-block and the gridded cell
list, every launch shape of the search, the coefficient adjoint around its
tiles, coefficients set from the host and from the device (GPU)."""
import numpy as np
import pytest

import mbx_oracle as mo
from mbx_b200 import system as msys, workloads
from mbx_b200.specs import SPECS
from mbx_b200.tables import load_fit

pytestmark = pytest.mark.gpu

E_REL = 1e-10
G_ABS = 1e-8
E_ABS_NMER = 1e-8   # one n-mer: its terms are up to 1e6 times their sum (test_gpu_parity)


# 1 dimer and no trimer; 1 trimer; a few; around one chunk of 384 n-mers (28
# waters have 378 dimers, 29 have 406); several chunks
@pytest.mark.parametrize("n", [2, 3, 9, 28, 29, 60])
def test_chunks_cut_by_pieces(n):
    ids, xyz = workloads.water_cluster(n, seed=n)
    s = msys.from_arrays(ids, xyz, None, 20.0, 20.0)
    ref = mo.OracleSystem(ids, xyz, None, 20.0, 20.0)
    for nb in (2, 3):
        e, er = (s.TwoBodyEnergy(True) if nb == 2 else s.ThreeBodyEnergy(True)), ref.energy(nb)
        assert abs(e - er) <= E_REL * abs(er) + E_ABS_NMER
        assert np.abs(s.GetRealGrads() - ref.real_grads()).max() <= G_ABS
        eo = s.TwoBodyEnergy(False) if nb == 2 else s.ThreeBodyEnergy(False)
        assert abs(eo - er) <= E_REL * abs(er) + E_ABS_NMER


# one block of 1024 threads builds the cell list, up to 640 members
@pytest.mark.parametrize("n", [639, 640, 641, 1023, 1024, 1025])
def test_search_around_one_block(n):
    edge = 39.44 * (n / 2048) ** (1 / 3)
    ids, xyz, box = workloads.water_box(12, n, edge, seed=n)
    s = msys.from_arrays(ids, xyz, box, 9.0, 7.0)
    o = xyz.reshape(-1, 9)[:, :3]
    d = o[:, None, :] - o[None, :, :]
    d -= edge * np.round(d / edge)
    i, j = np.nonzero(np.triu((d ** 2).sum(2) < 81.0, 1))
    assert np.array_equal(s.GetPairList(2, 9.0), np.stack([i, j], 1))


@pytest.mark.parametrize("box", ["wide", "narrow", "none"])
def test_search_launch_shapes(box):
    """wide: three or more cells per axis (one copy of every member); narrow:
    two cells (eight copies); none: no periodic boundaries.  The lists are the
    oracle's, for every launch shape."""
    if box == "none":
        ids, xyz = workloads.water_cluster(150, seed=4)
        b = None
    else:
        n = 700 if box == "wide" else 230
        ids, xyz, b = workloads.water_box(10 if box == "wide" else 7, n, 39.44 * (n / 2048) ** (1 / 3), seed=4)
    s = msys.from_arrays(ids, xyz, b, 9.0, 7.0)
    ref = mo.OracleSystem(ids, xyz, b, 9.0, 7.0)
    want = {nb: ref.top.nmers_to_input(ref.nmers(nb, 7.0)) for nb in (2, 3)}
    assert len(want[3]) > 1000
    for nb in (2, 3):
        assert np.array_equal(s.GetPairList(nb, 7.0), want[nb])
    for warps, unroll, threads in ((1, 1, 64), (1, 4, 256), (4, 1, 256), (4, 4, 64)):
        for nb in (2, 3):
            s._ctx.set_knobs(nb, nb_warps=warps, nb_unroll=unroll, tri_threads=threads)
            assert np.array_equal(s.GetPairList(nb, 7.0), want[nb])


def nmers(name, n, seed):
    rng = np.random.default_rng(seed)
    parts = []
    for k, m in enumerate(SPECS[name].monomers):
        v = rng.normal(size=(n, 3))
        r = rng.uniform(2.8, 5.0, size=n) * (k > 0)
        body = workloads.BODIES[m]() if m in workloads.BODIES else np.zeros((1, 3))
        parts.append(workloads.place(rng, body, v / np.linalg.norm(v, axis=1, keepdims=True) * r[:, None]))
    return np.ascontiguousarray(np.concatenate(parts, 1).reshape(n, -1))


# one n-mer; a tile of 8 and one more; several blocks; more than one chunk of
# 32768; one range of terms (mbpol2b), two (mbpol3b), half-monomials of degree
# 3 (h2oli2b); fewer terms than a warp's lanes times two (csh22b); few enough
# for one kernel (nana2b, hehe2b), with one block, two, and more n-mers than
# threads
@pytest.mark.parametrize("name,n", [("mbpol2b", 1), ("mbpol2b", 8), ("mbpol2b", 9), ("mbpol2b", 32769),
                                    ("mbpol3b", 1000), ("h2oli2b", 77), ("clh2o3b", 50), ("nana2b", 5),
                                    ("h2ona3b", 60), ("ch4ch42b", 20),
                                    ("nana2b", 128), ("nana2b", 129), ("nana2b", 40000), ("hehe2b", 300),
                                    ("csh22b", 33), ("csh22b", 33000)])
def test_adjoint_is_the_energy_per_coefficient(ctx, name, n):
    """The energy is linear in the coefficients: sum_k a_k dE/da_k = E; every
    dE/da_k is the oracle's sum over the terms in x; and the sums are made in
    the same order every time."""
    import torch
    x = torch.tensor(nmers(name, n, 5), device="cuda")
    w = torch.tensor(np.random.default_rng(6).uniform(-1, 1, n), device="cuda")
    a = load_fit(name)
    e = torch.empty(n, dtype=torch.float64, device="cuda")
    ctx.evaluate(name, x, None, None, e, grads=False)
    out = [torch.zeros(len(a), dtype=torch.float64, device="cuda") for _ in range(2)]
    for o in out:
        ctx.evaluate_dcoef(name, x, w, o)
    torch.cuda.synchronize()
    assert torch.equal(out[0], out[1])
    d = out[0].cpu().numpy()
    we = (w * e).cpu().numpy()
    # rounding of the products a_k d_k and of their sum, and of the energies
    bound = 64 * 2.0 ** -53 * np.abs(a * d).sum() + E_ABS_NMER * np.sqrt(n)
    assert abs((a * d).sum() - we.sum()) <= bound
    xyz, wn = x.cpu().numpy(), w.cpu().numpy()
    ref, size = np.zeros(len(a)), np.zeros(len(a))
    for b in range(0, n, 4096):
        per = wn[b:b + 4096, None] * mo.holder_dcoef(name, xyz[b:b + 4096])
        ref += per.sum(0)
        size += np.abs(per).sum(0)
    # The products in w that make up dE/da_k come to at most 5e3 times those in
    # x (the reference point of MB-pol 3b and the alkali 3b; 250 without one),
    # each rounded some 100 times: exponential, w, factors, sums
    assert np.all(np.abs(d - ref) <= 5e3 * 100 * 2.0 ** -53 * size)


@pytest.mark.parametrize("name", ["mbpol2b", "mbpol3b", "clh2o3b"])
def test_adjoint_of_weightless_nmers(ctx, name):
    """N-mers of weight 0 add nothing, whatever their coordinates: padding with
    all atoms at the origin has infinite variables."""
    x = nmers(name, 64, 11)
    w = np.random.default_rng(12).uniform(-1, 1, 64)
    alone = ctx.evaluate_dcoef(name, x, w)
    padded = ctx.evaluate_dcoef(name, np.concatenate([x, np.zeros_like(x)]), np.concatenate([w, np.zeros(64)]))
    size = np.abs(w[:, None] * mo.holder_dcoef(name, x)).sum(0)
    assert np.all(np.abs(padded - alone) <= 5e3 * 100 * 2.0 ** -53 * size)   # (sums in another order)


@pytest.mark.parametrize("name", ["mbpol2b", "mbpol3b", "h2ona3b", "ch4h2o3b", "co2co22b"])
def test_coefficients_from_host_and_device(ctx, name):
    import torch
    x = torch.tensor(nmers(name, 300, 7), device="cuda")
    a = load_fit(name) * np.random.default_rng(8).uniform(0.9, 1.1, SPECS[name].ncoef)

    def energies(coef, mixed):
        ctx.set_coefficients(name, coef)
        e, g = torch.empty(300, dtype=torch.float64, device="cuda"), torch.zeros_like(x)
        ctx.evaluate(name, x, g, None, e, mixed=mixed)
        torch.cuda.synchronize()
        return e, g

    for mixed in (False, True):
        fitted = energies(None, mixed)
        host = energies(a, mixed)
        device = energies(torch.tensor(a, device="cuda"), mixed)
        again = energies(None, mixed)
        assert not torch.equal(fitted[0], host[0])
        for p, q in ((host, device), (fitted, again)):
            assert torch.equal(p[0], q[0]) and torch.equal(p[1], q[1])


def test_operands_of_host_and_device_builder(ctx):
    """The tensor-core operands that mbx_set_coefficients builds on the device
    are the bytes mbx_qf_image builds on the host."""
    from mbx_b200 import capi
    fit = load_fit("mbpol3b")
    rng = np.random.default_rng(9)
    wide = fit * 10.0 ** rng.uniform(-9, 3, len(fit))   # parts of every size, subnormal ones among them
    some = np.where(rng.random(len(fit)) < 0.5, fit, 0.0)
    for a in (fit * rng.uniform(0.9, 1.1, len(fit)), wide, some, None):
        ctx.set_coefficients("mbpol3b", a)
        host, device = capi.qf_image("mbpol3b", a), ctx.qf_device_image("mbpol3b")
        assert host[0] == device[0]
        assert np.array_equal(host[1], device[1]) and host[2] == device[2]


def test_no_wait_refuses_what_it_cannot_give(ctx):
    """Host arrays, the mixed path, an energy sum and a virial are refused; the
    same call without them gives the energies."""
    import ctypes

    import torch
    from mbx_b200 import capi
    x = torch.tensor(nmers("mbpol2b", 40, 3), device="cuda")
    e = torch.zeros(40, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    sum_, vir = ctypes.c_double(), np.zeros(9)
    base = capi.MBX_NO_WAIT | capi.MBX_DEVICE_PTRS | capi.MBX_NO_GRADS

    def call(flags, virial=None, energy=None, xyz=x.data_ptr(), e_per=e.data_ptr()):
        return capi.lib().mbx_evaluate(ctx.h, b"mbpol2b", 40, xyz, None, virial, e_per, energy, flags)

    host = x.cpu().numpy()
    out = np.zeros(40)
    assert call(capi.MBX_NO_WAIT | capi.MBX_NO_GRADS, xyz=host.ctypes.data, e_per=out.ctypes.data) == 22
    assert call(base | capi.MBX_MIXED) == 22
    assert call(base, virial=vir.ctypes.data) == 22
    assert call(base, energy=ctypes.byref(sum_)) == 22
    assert not out.any() and not e.any()
    assert call(base) == 0
    torch.cuda.synchronize()
    ref = mo.holder_eval("mbpol2b", host, do_grads=False, per_nmer=True)[3]
    assert np.abs(e.cpu().numpy() - ref).max() <= E_ABS_NMER
