"""The spins of a growth step are spread four to a lane and its directions over the first lanes of a warp: trial counts at
the edges of those against the exact ideal-gas Rosenbluth weight of butane and the exact mean of its torsion cosine.

Any trial count gives an unbiased weight: the mean of 100,000 growths is within 5 standard errors of the exact value (one
run in 1.7 million outside for each of the six), and so is the weighted mean of the cosine."""

import math

import numpy as np
import pytest

from raspa3_b200 import native
from raspa3_b200.alkane import AlkaneChain, alkane_forcefield
from raspa3_b200.gcmc import beta_of
from test_oracle_alkane import butane_exact

pytestmark = pytest.mark.gpu
BETA = beta_of(300.0)


@pytest.mark.parametrize("directions,spins", [(1, 1), (1, 128), (16, 5), (2, 3), (16, 127), (15, 4)])
def test_trial_counts(directions, spins):
    ctx = native.Context(0)
    ff = alkane_forcefield()
    chain = AlkaneChain(4, n_directions=directions, n_torsion=spins)
    mean, w, _, cosine = native.alkane_grow_vacuum(ctx, ff, chain, BETA, 100000, seed=11, details=True)
    exact, exact_cosine = butane_exact(AlkaneChain(4), ff)
    se = w.std(ddof=1) / math.sqrt(len(w))
    assert abs(mean - exact) <= 5 * se, (mean, exact, se)
    x = w * (cosine[:, 0] - exact_cosine)  # zero mean, whatever the trial counts
    assert abs(x.mean()) <= 5 * x.std(ddof=1) / math.sqrt(len(x))
    ctx.close()
