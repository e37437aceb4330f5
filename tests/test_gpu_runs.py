"""Blocks of the stencil kernels that take many (tile, shot) items (B200).

A small grid of six (or twelve) tiles with far more shots than the device has
blocks for: every block takes a run of shots of a tile, so that the stages of
its ring are refilled, their barriers change phase several times and the sums
of a run are formed.  All modes against the FP64 oracle, with the tolerances
of tests/test_gpu_parity.py (traces 1e-5, gradients 2e-5 times
|pred| / |pred - obs|).
"""
import functools

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

NZ, NX, PAD, DX, DT, FC, NT, NS = 20, 120, 8, 10.0, 1.0e-3, 25.0, 40, 240


def _rel(a, b):
    a = np.asarray(a, np.float64); b = np.asarray(b, np.float64)
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


@functools.lru_cache(maxsize=None)
def _case(fd, fs):
    rng = np.random.default_rng(fd)
    zz = np.arange(NZ)[:, None] / NZ
    vp = 2300.0 + 700.0 * zz + 60.0 * rng.standard_normal((NZ, NX))
    vs, rho = vp / 1.8, 1900.0 + 200.0 * zz + 20.0 * rng.standard_normal((NZ, NX))
    rx = np.arange(0, NX, 6, dtype=np.int32)
    rz = np.where(np.arange(len(rx)) % 2 == 0, 1, NZ - 2).astype(np.int32)
    sx, sz = rng.integers(0, NX, NS), rng.integers(0, NZ, NS)
    types = [("force", "moment")[k % 2] for k in range(NS)]
    wav = O.ricker(np.arange(NT) * DT, FC, 0.5 / FC) * 1e9
    geo = dict(rec_x=rx, rec_z=rz, nx_dom=NX, nz_dom=NZ, dx=DX, dz=DX, dt=DT, nt=NT, fc=FC, pad=PAD, fd_order=fd,
               free_surface=fs, d0_f32=True)
    ref = O.forward_batch(vs, vp, rho, sx, sz, types, src_wavelet=wav, **geo)
    obs = O.forward_batch(vs * 1.03, vp, rho, sx, sz, types, src_wavelet=wav, **geo)[:, 1]
    kw = dict(Vs=vs, Vp=vp, rho=rho, src_x=sx, src_z=sz, src_wavelet=wav, observed=obs, src_types=types, component=1,
              scale=1.0, invert="all", **geo)
    exact, loss = O.compute_gradient("ad", **kw)
    imaging, _ = O.compute_gradient("adjoint", **kw)
    return (vs, vp, rho), (rx, rz), (sx, sz, types, wav.astype(np.float32)), ref, obs, exact, imaging, loss


def _solver(fd, fs, **kw):
    from stfwi_b200 import Solver
    model, rec, shots = _case(fd, fs)[:3]
    S = Solver(NZ, NX, DX, DX, DT, NT, FC, PAD, len(rec[0]), NS, fd_order=fd, free_surface=fs, **kw)
    S.set_receivers(*rec)
    S.set_shots(*shots)
    S.set_model(*model)
    return S


@pytest.mark.parametrize("tiles", [(16, 16), (8, 8)])
@pytest.mark.parametrize("fd,fs", [(2, False), (4, True), (8, True)])
def test_runs_of_shots_vs_oracle(fd, fs, tiles):
    ref, obs, exact, imaging, loss = _case(fd, fs)[3:]
    S = _solver(fd, fs, density=True, shot_group=7)
    S.set_tile_rows(*tiles)
    S.forward(store=True)
    rec = S.records()
    assert max(_rel(rec[:, c], ref[:, c]) for c in range(4)) < 1e-5
    mis = S.misfit(obs.astype(np.float32), 1, 1.0)
    tol = 2e-5 * max(float(np.linalg.norm(rec[:, 1]) / np.linalg.norm(rec[:, 1] - obs)), 1.0)
    g = S.gradient(exact=True, imaging=True)
    S.close()
    errs = {"misfit": abs(mis.sum() / loss - 1)}
    for k, name in enumerate(("vs", "vp", "rho")):
        errs["exact_" + name] = _rel(g["exact"][k], exact[k])
        errs["img_" + name] = _rel(g["imaging"][k], imaging[k])
    assert all(e < tol for e in errs.values()), (tol, errs)


@pytest.mark.parametrize("group", [0, 1, 7])
@pytest.mark.parametrize("density", [False, True])
def test_gradients_repeat_bit_for_bit(group, density):
    """Every block's FP32 sums go to FP64 planes of its own, step by step: a
    second pass, and a pass in another number of chains, gives the same bits,
    for the default runs, for runs of one shot and for long ones."""
    fd, fs = 8, True
    obs = _case(fd, fs)[4].astype(np.float32)
    S = _solver(fd, fs, density=density, shot_group=group)
    out = []
    for chains in (2, 2, 1, 3, 4):
        S.set_chains(chains)
        S.forward(store=True)
        S.misfit(obs, 1, 1.0)
        g = S.gradient(exact=True, imaging=True)
        out.append((S.records(), g["exact"], g["imaging"]))
    S.close()
    for k in range(1, len(out)):
        for a, b in zip(out[0], out[k]):
            assert np.array_equal(a, b), k
