"""Shapes at which the kernels of a PCG pass change: the bra-ket's 32 x 32, 64 x 64
and 112 x 64 tiles (64 | 65 systems, 64 | 65 and 112 | 113 projectors), odd
projector counts (rows of 8, split rows of 2 x 64 and more), one and several
buckets of the captured loop, the step kernel's clusters of 1 to 8 CTAs (few
systems of many plane waves), and boxes that run the plane phases with radices
taken at run time.  Converged solves (tr2 far below the production threshold) in
FP64 against the oracle at the tolerance of the other parity tests (1e-10)."""
import dataclasses

import numpy as np
import pytest

from oracle import west_oracle as O
from west_b200.system import SystemSpec, build_system, perturbations

pytestmark = pytest.mark.gpu


def _solve(s, dvg, graphs=True):
    from west_b200.wstat import ResponseOperator
    op = ResponseOperator(s, n_dfpt_maxiter=400, verbose=False)
    op.set_graphs(graphs)
    dng = np.zeros_like(dvg, order="F")
    ierr = op.apply_operator(dvg.shape[1], dvg, dng, 1e-20, 1)
    op.close()
    return dng, ierr


def _check(s, m):
    dvg = perturbations(s, m, seed=m)
    k = min(m, 2)                                   # the oracle takes the first and the last
    pick = [0, m - 1][:k]
    ref, rerr = O.apply_operator(s, np.asfortranarray(dvg[:, pick]), 1e-20, maxiter=400)
    assert (rerr == 0).all()
    got, ierr = _solve(s, dvg)
    assert (ierr == 0).all()
    assert np.linalg.norm(got[:, pick] - ref) / np.linalg.norm(ref) < 1e-10
    eager, _ = _solve(s, dvg, graphs=False)
    assert np.linalg.norm(got - eager) / np.linalg.norm(eager) < 1e-10


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


@pytest.mark.parametrize("L,ecut,nr", [(13.0, 12.0, 32), (15.0, 20.0, 48), (17.0, 25.0, 60)])   # clusters of 2, 4, 8
def test_step_clusters(L, ecut, nr):
    _check(build_system(SystemSpec(L=L, ecutwfc=ecut, nr=nr, natoms=2, nbnd_occ=3, proj="s", seed=4), "cuda"), 2)


@pytest.mark.parametrize("L,ecut,nr", [
    ((12.0, 13.0, 11.0), 10.0, (27, 30, 25)),       # radices 3 to 9, odd edges
    ((16.0, 18.0, 21.0), 10.0, (45, 54, 60)),       # more room than the sphere needs
    ((20.0, 9.0, 9.0), 16.0, (75, 35, 35)),         # radices 15, 7
    ((9.0, 28.0, 9.0), 16.0, (36, 112, 40)),        # radix 16
    ((10.0, 10.0, 30.0), 10.0, (42, 45, 125)),      # a z edge without a split
])
def test_runtime_planes(L, ecut, nr):
    _check(build_system(SystemSpec(L=L, ecutwfc=ecut, nr=nr, natoms=2, nbnd_occ=3, proj="sp", seed=5), "cuda"), 3)
