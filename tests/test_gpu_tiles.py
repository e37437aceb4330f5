"""Sizes at the edges of the stencil kernels' tiles, strips and image bands (B200).

Traces, source adjoint and the exact gradient against the FP64 oracle on grids
whose padded size is just below, at and above whole tiles (64 columns, 8 or 16
rows), with odd rows, C-PML strips from the stencil's own reach to wider than
a tile, grids whose left and right bands meet, and sources and receivers on
the outermost physical cells and inside the strips.  Tolerances: FP32 against
FP64 as in tests/test_gpu_parity.py (traces and source adjoint 1e-5, gradients
2e-5 times |pred| / |pred - obs|).
"""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _rel(a, b):
    a = np.asarray(a, np.float64); b = np.asarray(b, np.float64)
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


# (nz, nx, pad, fd, free surface, shots, tile rows)
CASES = [
    (24, 48, 8, 8, True, 1, (16, 16)),       # padded 32 x 64: whole tiles, one column of tiles
    (25, 47, 8, 8, False, 2, (16, 8)),       # padded 41 x 63
    (23, 49, 8, 4, True, 2, (8, 16)),        # padded 31 x 65: a tile of one column
    (40, 113, 8, 8, True, 9, (16, 16)),      # padded 48 x 129: bands apart, more shots than a block's run
    (41, 111, 4, 8, False, 3, (8, 8)),       # the thinnest strip of FD 8, odd width
    (9, 12, 1, 2, True, 2, (16, 16)),        # the thinnest strip of FD 2, a grid below one tile
    (9, 11, 4, 8, False, 3, (16, 16)),       # masks of both edges overlap
    (30, 70, 66, 4, True, 2, (16, 16)),      # a strip wider than a tile
    (33, 190, 13, 8, True, 4, (16, 16)),     # odd strip: history by plain loads
]


@pytest.mark.parametrize("nz,nx,pad,fd,fs,ns,tiles", CASES)
def test_tile_edges_vs_oracle(nz, nx, pad, fd, fs, ns, tiles):
    from stfwi_b200 import Solver
    nt, dx, dt, fc = 70, 10.0, 1.0e-3, 25.0
    rng = np.random.default_rng(nz * 1000 + nx)
    zz = np.arange(nz)[:, None] / nz
    vp = 2300.0 + 700.0 * zz + 60.0 * rng.standard_normal((nz, nx))
    vs, rho = vp / 1.8, 1900.0 + 200.0 * zz + 20.0 * rng.standard_normal((nz, nx))
    # outermost physical cells and strip cells (physical indices below 0 and beyond the model)
    rx = np.array([0, 1, nx // 2, nx - 1, -1, nx, nx // 2, min(61, nx - 1)], dtype=np.int32)
    rz = np.array([0, nz - 1, nz // 2, 0, nz // 3, nz // 2, nz, 1], dtype=np.int32)
    sx = np.linspace(0, nx - 1, ns).astype(np.int64)
    sz = np.array([(0, nz - 1, nz // 2)[k % 3] for k in range(ns)])
    types = [("force", "moment")[k % 2] for k in range(ns)]
    wav = O.ricker(np.arange(nt) * dt, fc, 1.2 / fc) * 1e9
    geo = dict(rec_x=rx, rec_z=rz, nx_dom=nx, nz_dom=nz, dx=dx, dz=dx, dt=dt, nt=nt, fc=fc, pad=pad, fd_order=fd,
               free_surface=fs, d0_f32=True)
    ref = O.forward_batch(vs, vp, rho, sx, sz, types, src_wavelet=wav, **geo)
    obs = O.forward_batch(vs * 1.03, vp, rho, sx, sz, types, src_wavelet=wav, **geo)[:, 1]
    (g_vs, g_vp, g_rho), loss = O.compute_gradient("ad", Vs=vs, Vp=vp, rho=rho, src_x=sx, src_z=sz, src_wavelet=wav,
                                                   observed=obs, src_types=types, component=1, scale=1.0,
                                                   invert="all", **geo)
    S = Solver(nz, nx, dx, dx, dt, nt, fc, pad, len(rx), ns, fd_order=fd, free_surface=fs, density=True)
    S.set_tile_rows(*tiles)
    S.set_receivers(rx, rz)
    S.set_shots(sx, sz, types, wav.astype(np.float32))
    S.set_model(vs, vp, rho)
    S.forward(store=True)
    rec = S.records()
    for k in range(ns):
        for c in range(4):
            assert _rel(rec[k, c], ref[k, c]) < 1e-5, (k, c, _rel(rec[k, c], ref[k, c]))
    mis = S.misfit(obs.astype(np.float32), 1, 1.0)
    tol = 2e-5 * max(float(np.linalg.norm(rec[:, 1]) / np.linalg.norm(rec[:, 1] - obs)), 1.0)
    g = S.gradient(exact=True)["exact"]
    errs = {"misfit": abs(mis.sum() / loss - 1), "vs": _rel(g[0], g_vs), "vp": _rel(g[1], g_vp), "rho": _rel(g[2], g_rho)}
    assert all(e < tol for e in errs.values()), (tol, errs)
    # the source adjoint of random receiver sources on all four components
    ys = rng.standard_normal((ns, 4, nt, len(rx)))
    S.set_adjoint_sources(ys.astype(np.float32))
    src = S.gradient(exact=False, src=True)["src"]
    for k in range(ns):
        a = O.adjoint(vs, vp, rho, sx[k], sz[k], rx, rz, nx, nz, dx, dx, dt, nt, fc, pad, *ys[k], fd_order=fd,
                      free_surface=fs, src_type=types[k], d0_f32=True)
        assert _rel(src[k], a["src"]) < 1e-5, (k, _rel(src[k], a["src"]))
    S.close()
