"""Records put in place as they are encoded: one runner takes populations that grow, shrink and change their kind from
call to call, so that what the call before left room for is too much, just enough or too little."""
import numpy as np
import pytest
import torch

from secant_b200 import abi, programs as P
from secant_b200.runner import Runner

pytestmark = pytest.mark.gpu


def populations():
    plain = lambda n, tokens, seed: P.random_population(seed, n, tokens, 3, 4, 1.0, ops=P.ARITHMETIC_OPS)  # noqa: E731
    toggled = lambda n, tokens, seed: P.random_population(seed, n, tokens, 3, 4, 1.0, toggle_bits=3, ops=P.ARITHMETIC_OPS)  # noqa: E731
    literals = P.PackedPrograms([P.lit(0.001 * i) + P.lit(0.5 + i) + P.col(0) + P.op("MUL") + P.op("ADD") + P.RET for i in range(200)])
    affine = P.PackedPrograms([P.affine(i % 4, 1.0 + i, 0.5) + P.col(1) + P.op("MUL") + P.RET for i in range(200)])
    return [plain(300, 8, 1), plain(300, 8, 2), plain(40, 8, 3), plain(300, 32, 4), plain(2000, 20, 5), toggled(300, 24, 6), toggled(1000, 24, 7),
            plain(1, 4, 8), literals, affine, plain(4097, 12, 9), plain(9000, 12, 10), plain(130, 30, 11)]


@pytest.mark.parametrize("workers", [1, 4])
def test_populations_of_changing_size_and_kind(cuda, workers):
    rows, banks = 65, 3
    rng = np.random.default_rng(2)
    dev = lambda *shape: torch.tensor(rng.standard_normal(shape).astype(np.float32), device="cuda")  # noqa: E731
    x, y, table = dev(3, rows), dev(1, rows), dev(banks, 4)
    with Runner(abi.SHAPE_TOGGLE_SSE, 3, 1, 4, workers=workers, streams=2) as rn:
        for pop in populations() * 2:
            scores = []
            for run in (rn.run, None):
                out = torch.full((len(pop.asts), 1, banks << 3), 5.0, device="cuda")
                torch.cuda.synchronize()
                request = rn.toggle_request(pop, x, y, table, banks, 3, out)
                if run:
                    run(request)
                else:
                    resident = rn.population(pop, 3)              # encoded and packed by one thread
                    resident.run(request)
                    resident.destroy()
                scores.append(out.cpu().numpy())
            assert np.array_equal(scores[0].view(np.uint32), scores[1].view(np.uint32))
