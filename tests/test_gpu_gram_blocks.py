"""Cohort statistics where the kernels' blocks end: eight features to a block, two targets with it and eight to a block beyond
them, 256 rows a step of a CTA and eight CTAs to a range."""
import numpy as np
import pytest
import torch

import support as S
from secant_b200 import abi, programs as P
from secant_b200.runner import Runner

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("programs,cohort", [(1, 1), (8, 8), (15, 8), (9, 9), (33, 16), (17, 17), (47, 32)])
@pytest.mark.parametrize("rows,targets", [(1, 1), (2, 2), (255, 3), (2047, 2), (2049, 10), (4353, 11)])
def test_every_statistic_is_written_once(cuda, programs, cohort, rows, targets):
    ops = [(P.op("ADD"), 2), (P.op("SUB"), 2), (P.op("MUL"), 2), (P.op("COS"), 1)]
    pop = P.random_population(7 + programs, programs, 9, 3, ops=ops)
    x = np.stack([P.uniform(8, c, rows, -1, 1) for c in range(3)])
    y = np.stack([P.normal(9, t, rows) for t in range(targets)])
    lead = rows + 3                                                  # targets that start at every alignment
    padded = torch.zeros((targets, lead), device="cuda")
    padded[:, :rows] = torch.tensor(y, device="cuda")
    with Runner(abi.SHAPE_GRAM_STATS, 3, targets, num_kernels=4, asts_per_kernel=cohort, workers=2, streams=2) as rn:
        width = cohort * (1 + cohort + targets)
        out = torch.full((-(-programs // cohort), width), 7.0, device="cuda")
        data = torch.tensor(x, device="cuda")
        torch.cuda.synchronize()
        request = rn.static_request(pop, data, padded[:, :rows], out)
        request.targets.leading_dimension, request.targets.num_elements = lead, padded.numel()
        rn.run(request)
        got = out.cpu().numpy()
    code, _, want = S.oracle_gram_stats(pop, x, y, cohort)
    assert code == 0
    # a sum is at most rows / 2,048 + 18 additions deep, products are rounded once: 22 x 2^-24 of the terms' magnitudes,
    # which the largest statistic of a cohort (a sum of squares) bounds to within the cohort's spread, and the oracle's inputs
    # are the same numbers
    assert np.all(np.abs(got - want) <= 2e-5 * (np.abs(want).max(axis=1, keepdims=True) + 1.0))
