"""The host pipeline's pieces and launch order: a run's scores equal, bit for bit, those of the same
programs made resident (one piece), at population sizes around the edges of a piece, of the sort and
of a batch."""
import numpy as np
import pytest
import torch

from secant_b200 import abi, programs as P
from secant_b200.runner import Runner

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("programs", [1, 16, 17, 129, 512, 513, 4096, 4097, 16385])
def test_every_program_lands_in_its_place(cuda, programs):
    base = P.random_population(7, min(programs, 1500), 16, 3, 4, 1.0)
    pop = P.PackedPrograms([base.asts[i % len(base.asts)] for i in range(programs)], base.routines)
    x = torch.tensor(np.stack([P.uniform(8, c, 77, -1, 1) for c in range(3)]), device="cuda")
    y = torch.tensor(np.stack([P.normal(9, 0, 77)]), device="cuda")
    banks = torch.tensor(np.stack([P.normal(10, b, 4) for b in range(3)]), device="cuda")
    with Runner(abi.SHAPE_TOGGLE_SSE, 3, 1, 4, workers=3, streams=2) as rn:
        out = torch.full((programs, 1, 3), 5.0, device="cuda")
        torch.cuda.synchronize()
        request = rn.toggle_request(pop, x, y, banks, 3, 0, out)
        rn.run(request)
        got = out.cpu().numpy()
        resident = rn.population(pop, 0)
        out.fill_(6.0)
        torch.cuda.synchronize()
        resident.run(request)
        want = out.cpu().numpy()
        resident.destroy()
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
    for first in range(len(base.asts), programs, len(base.asts)):      # repeated programs score alike
        n = min(len(base.asts), programs - first)
        assert np.array_equal(got[first:first + n].view(np.uint32), got[:n].view(np.uint32))
