"""Shapes at which the kernels of a PCG pass change: row tiles of the bra-ket (full,
even and ragged splits into 32, 5,634 and 6,144 projectors in its reduction), column
tiles, one and several buckets of the captured loop (64 | 65 systems), the step kernel's CTAs of 256, 512 and 1,024 threads
and clusters of four, and boxes that run the plane phases with radices taken at run
time.  Converged solves (tr2 far below the production threshold) against the oracle
at the tolerances of the other parity tests (1e-10, mixed form 1e-7)."""
import dataclasses

import numpy as np
import pytest

from oracle import west_oracle as O
from west_b200.system import SystemSpec, build_system, perturbations

pytestmark = pytest.mark.gpu


def _solve(s, dvg, graphs=True, form="fp64"):
    from west_b200.wstat import ResponseOperator
    op = ResponseOperator(s, n_dfpt_maxiter=400, verbose=False)
    op.set_graphs(graphs)
    op.set_precision(form)
    dng = np.zeros_like(dvg, order="F")
    ierr = op.apply_operator(dvg.shape[1], dvg, dng, 1e-20 if form == "fp64" else 1e-14, 1)
    op.close()
    return dng, ierr


def _check(s, m, form="fp64"):
    tol = 1e-10 if form == "fp64" else 1e-7
    dvg = perturbations(s, m, seed=m)
    k = min(m, 2)                                   # the oracle takes the first and the last
    pick = [0, m - 1][:k]
    ref, rerr = O.apply_operator(s, np.asfortranarray(dvg[:, pick]), 1e-20, maxiter=400)
    assert (rerr == 0).all()
    got, ierr = _solve(s, dvg, form=form)
    assert (ierr == 0).all()
    assert np.linalg.norm(got[:, pick] - ref) / np.linalg.norm(ref) < tol
    eager, _ = _solve(s, dvg, graphs=False, form=form)
    assert np.linalg.norm(got - eager) / np.linalg.norm(eager) < tol


@pytest.mark.parametrize("m", [1, 11, 21, 22, 43, 50])          # 3 bands: 3 to 150 systems
def test_system_counts(tiny, m):
    _check(tiny, m)


@pytest.mark.parametrize("natoms,nbnd", [(15, 4), (14, 9), (27, 4), (27, 5), (50, 8)])   # 64, 65, 112, 113, 208 projectors
def test_projector_counts(natoms, nbnd):
    s = build_system(SystemSpec(L=12.0, ecutwfc=8.0, nr=24, natoms=natoms, nbnd_occ=nbnd, proj="sp", Z=2.0,
                                dion=0.2, seed=3), "cuda")
    assert s.nkb + s.nbnd_occ in (64, 65, 112, 113, 208)
    _check(s, 17)


@pytest.mark.parametrize("total", [5634, 6144])
def test_reduction_of_many_projectors(tiny, total):
    """Projectors and bands whose sums take all of the 48 KB that the reduction has for
    them: zero projectors before tiny's own leave its response as it is."""
    s = tiny
    nkb = total - s.nbnd_occ
    vkb = np.zeros((s.npw, nkb), dtype=np.complex128, order="F")
    vkb[:, nkb - s.nkb:] = s.vkb
    deeq = np.zeros((nkb, nkb), order="F")
    deeq[nkb - s.nkb:, nkb - s.nkb:] = s.deeq
    dvg = perturbations(s, 2, seed=1)
    ref, _ = O.apply_operator(s, dvg, 1e-20, maxiter=400)
    got, ierr = _solve(dataclasses.replace(s, vkb=vkb, deeq=deeq), dvg)
    assert (ierr == 0).all()
    assert np.linalg.norm(got - ref) / np.linalg.norm(ref) < 1e-10


# plane waves up to 1,024, up to 4,095, and more: one CTA of 256 or 512 threads, clusters of four
_STEP_CELLS = [(13.0, 12.0, 32, 0, 1024), (15.0, 18.0, 45, 1025, 4095), (17.0, 25.0, 60, 4096, 10 ** 6)]


def _step_cell(L, ecut, nr, lo, hi):
    s = build_system(SystemSpec(L=L, ecutwfc=ecut, nr=nr, natoms=2, nbnd_occ=3, proj="s", seed=4), "cuda")
    assert lo <= s.npw <= hi
    return s


@pytest.mark.parametrize("form", ["fp64", "mixed"])
@pytest.mark.parametrize("m", [2, 23])                          # 6 systems, and 69: in the last cell 1,024 threads (FP64), 512 (mixed)
@pytest.mark.parametrize("cell", _STEP_CELLS)
def test_step_shapes(cell, m, form):
    _check(_step_cell(*cell), m, form)


@pytest.mark.parametrize("form", ["fp64", "mixed"])
@pytest.mark.parametrize("L,nr", [(25.0, 80), (30.0, 108)])     # clusters of 2 and 4 in FP64, 1 and 2 in FP32
def test_step_clusters_of_large_cells(L, nr, form):
    """66 systems, whose vectors pass L2 with one CTA each, against the same
    perturbations one by one (clusters of four)."""
    s = build_system(SystemSpec(L=L, ecutwfc=25.0, nr=nr, natoms=2, nbnd_occ=3, proj="s", seed=4), "cuda")
    assert s.npw > 16000
    dvg = perturbations(s, 22, seed=1)
    got, ierr = _solve(s, dvg, form=form)
    assert (ierr == 0).all()
    for p in (0, 21):
        one, _ = _solve(s, np.asfortranarray(dvg[:, p:p + 1]), form=form)
        assert np.linalg.norm(got[:, p] - one[:, 0]) / np.linalg.norm(one) < (1e-10 if form == "fp64" else 1e-7)


@pytest.mark.parametrize("form", ["fp64", "mixed"])
@pytest.mark.parametrize("cell", _STEP_CELLS)
def test_bits_do_not_depend_on_earlier_calls(cell, form):
    """A call gives the same bits first on its context, after larger calls (whose
    workspace its captured loop then has) and eagerly, and up to 64 systems through the
    allocation-free entry point where they fit it."""
    import ctypes
    import torch
    from west_b200 import lib as L
    from west_b200.wstat import ResponseOperator
    s = _step_cell(*cell)
    dvg = perturbations(s, 43, seed=2)

    def op():
        o = ResponseOperator(s, verbose=False)
        o.set_precision(form)
        o.set_autotune(form == "fp64")                          # the mixed form times shapes, per context
        return o

    def run(o, m):
        dng = np.zeros((s.npw, m), dtype=np.complex128, order="F")
        o.apply_operator(m, np.asfortranarray(dvg[:, :m]), dng, 1e-10, 1)
        return dng

    grown, eager = op(), op()
    eager.set_graphs(False)
    run(grown, 43)
    for m in (1, 22, 43, 1):
        first = run(op(), m)
        assert np.array_equal(run(grown, m), first), m
        assert np.array_equal(run(eager, m), first), m
    if form == "fp64":
        o, dv = op(), torch.from_numpy(np.ascontiguousarray(dvg[:, :1].T)).cuda()
        out = torch.zeros_like(dv)
        ierr = ctypes.c_int(-1)
        rc = L.load().wb_apply_operator_device_noalloc(o._ctx, 1, dv.data_ptr(), s.npw, out.data_ptr(), s.npw, 1e-10, 1,
                                                       ctypes.addressof(ierr))
        assert rc == 0 and ierr.value == 0
        assert np.array_equal(out.cpu().numpy().T, run(op(), 1))


@pytest.mark.parametrize("L,ecut,nr", [
    ((12.0, 13.0, 11.0), 10.0, (27, 30, 25)),       # radices 3 to 9, odd edges
    ((16.0, 18.0, 21.0), 10.0, (45, 54, 60)),       # more room than the sphere needs
    ((20.0, 9.0, 9.0), 16.0, (75, 35, 35)),         # radices 15, 7
    ((9.0, 28.0, 9.0), 16.0, (36, 112, 40)),        # radix 16
    ((10.0, 10.0, 30.0), 10.0, (42, 45, 125)),      # a z edge without a split
])
def test_runtime_planes(L, ecut, nr):
    _check(build_system(SystemSpec(L=L, ecutwfc=ecut, nr=nr, natoms=2, nbnd_occ=3, proj="sp", seed=5), "cuda"), 3)
