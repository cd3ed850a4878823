"""FP64 products of a few contraction steps (splits whose last slices are short
or empty) and the dictionary-learning tiles of at most 32 columns."""
import numpy as np
import pytest

import oracle
import rwig_b200 as rw
from rwig_b200 import synth
from tests.test_gpu_dgemm import _run
from tests.util import PARITY_TOL, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("trans", [0, 1])
@pytest.mark.parametrize("Mo,Kd,S", [(40, 31, 5), (64, 33, 32), (65, 64, 33), (70, 127, 7), (64, 128, 64), (63, 129, 30),
                                     (500, 161, 20)])
def test_short_slices(trans, Mo, Kd, S):
    g = np.random.default_rng(Mo + 3 * Kd + S)
    K = g.standard_normal((Kd, Mo) if trans else (Mo, Kd))
    X = g.standard_normal((Kd, S))
    ref = (K.T if trans else K) @ X
    assert np.abs(_run(K, X, trans) - ref).max() <= 1e-12 * max(1.0, np.abs(ref).max()) * np.sqrt(Kd)


# whole documents in tiles of 32 (S = 4, 6, 31, 32), of 64 (33; 20 where 32 pads
# more), a single document, and enough columns for the wide kernel
@pytest.mark.parametrize("N,D,S", [(70, 8, 4), (129, 11, 6), (65, 3, 31), (64, 2, 32), (90, 3, 33), (200, 16, 20),
                                   (61, 1, 6), (1000, 65, 20)])
def test_document_tiles(N, D, S):
    Y, C, A0, L0 = synth.wdl_config(V=N, M=D, S=S, dim=8, salt=N + D + S)
    A, W = oracle.col_softmax(A0), oracle.col_softmax(L0)
    K = np.asfortranarray(np.exp(-C / 0.1))
    ref_gA, ref_gl = oracle.wdl_batch_grad(A, W, Y, K, 3)
    gA, gl = rw.wdl_batch_grad(A, W, Y, K, 0.1, 3, mode=0)
    assert rel_err(gA, ref_gA) <= PARITY_TOL
    assert rel_err(gl, ref_gl) <= PARITY_TOL
