"""1- and 2-RDMs summed per label on the device (csrc/rdm.cu) against the oracle: fewer labels and
columns than a block, labels of one single, unequal spins, a wide orbital space."""
import itertools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = {  # norb, (alpha electrons, strings), (beta electrons, strings)
    "full6": (6, (3, 20), (3, 20)),
    "unequal": (12, (4, 70), (3, 41)),
    "wide": (40, (3, 60), (2, 33)),        # 1,600 columns of label sums: several blocks of threads
    "one_string": (8, (3, 1), (4, 30)),    # no alpha singles at all
    # 8 orbitals: doubles are summed per label from 257 of them, placed one by one below
    "summed_and_placed": (8, (4, 40), (4, 18)),
}


def _strings(norb, n, count, seed):
    idx = np.array(list(itertools.combinations(range(norb), n)), np.int64)
    score = idx.sum(axis=1) + 2.0 * np.random.default_rng(seed).gumbel(size=len(idx))
    score[0] = -np.inf
    return np.sort((np.int64(1) << idx[np.argsort(score, kind="stable")[:count]]).sum(axis=1).astype(np.uint64))


@pytest.mark.parametrize("name", sorted(CASES))
def test_rdm_label_sums_against_oracle(name):
    import pyoracle
    import sbd_tpb
    import synth
    norb, (ea, na), (eb, nb) = CASES[name]
    h1, eri, core = synth.synthetic_hamiltonian(norb, seed=3)
    prob = sbd_tpb.Problem(norb=norb, nelec=ea + eb, core=core, h1=h1, eri_packed=eri,
                           astr=_strings(norb, ea, na, 1), bstr=_strings(norb, eb, nb, 2))
    W = np.random.default_rng(4).normal(size=prob.ndet)
    W /= np.linalg.norm(W)
    ham = pyoracle.Hamiltonian.from_arrays(norb, prob.nelec, core, h1, eri)
    ref1, ref2 = pyoracle.System(ham, prob.astr, prob.bstr).rdm(W)[:2]
    h = sbd_tpb.Handle(0)
    h.set_problem(prob)
    one, two = h.rdm(W)
    h.close()
    # FP64 sums of at most a few thousand products of a normalised vector
    assert np.max(np.abs(one - np.asarray(ref1).ravel())) < 1e-13
    assert np.max(np.abs(two - np.asarray(ref2).ravel())) < 1e-13
