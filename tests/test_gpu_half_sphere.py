"""Half spheres in another order than QE's: any choice of +G or -G per pair is a
Gamma half sphere (psi(-G) = conj psi(G)).  A stick pair whose coefficients then
are not one run of one side sends the compiled boxes' z passes to their table
form, which must give the run form's results: the response of the flipped system
is the conjugate of the oracle's at the flipped G.  Converged solves, 1e-10 as in
the other parity tests; the mixed form 1e-7."""
import dataclasses

import numpy as np
import pytest

from oracle import west_oracle as O
from west_b200.system import SystemSpec, build_system, perturbations

pytestmark = pytest.mark.gpu


def _flip(a, mask):
    a = a.copy()
    a[mask] = a[mask].conj()
    return np.asfortranarray(a)


@pytest.mark.parametrize("share", [0.5, 0.02])                  # most pairs mixed; few
@pytest.mark.parametrize("L,ecut,nr", [(10.0, 8.0, 24), (14.0, 12.0, 40), ((10.0, 11.0, 12.0), 8.0, (27, 25, 30))])
def test_flipped_half(L, ecut, nr, share):
    from west_b200.wstat import ResponseOperator
    s = build_system(SystemSpec(L=L, ecutwfc=ecut, nr=nr, natoms=2, nbnd_occ=3, proj="sp", seed=8), "cuda")
    mask = np.random.default_rng(1).random(s.npw) < share
    mask[0] = False
    f = dataclasses.replace(s, mill=np.where(mask[:, None], -s.mill, s.mill), nl=np.where(mask, s.nlm, s.nl),
                            nlm=np.where(mask, s.nl, s.nlm), evc=_flip(s.evc, mask), vkb=_flip(s.vkb, mask))
    dvg = perturbations(s, 3, seed=6)
    ref, _ = O.apply_operator(s, dvg, 1e-20, maxiter=400)
    for form, tol in (("fp64", 1e-10), ("mixed", 1e-7)):
        op = ResponseOperator(f, n_dfpt_maxiter=400, verbose=False)
        op.set_precision(form)
        dng = np.zeros_like(dvg, order="F")
        ierr = op.apply_operator(3, _flip(dvg, mask), dng, 1e-20 if form == "fp64" else 1e-14, 1)
        op.close()
        assert (ierr == 0).all()
        assert np.linalg.norm(_flip(dng, mask) - ref) / np.linalg.norm(ref) < tol
