"""The refinement's GMRES issues a step before it has read the one before: not where that one will be given up."""
import numpy as np
import pytest

from test_gpu_parity import small  # noqa: F401 (the fixture)

pytestmark = pytest.mark.gpu

torch = pytest.importorskip('torch')


@pytest.mark.parametrize('rule,steps', [(dict(give_up=(10, 0.05)), 10), (dict(stagnate=(10, 0.5)), 10),
                                        (dict(stall=(4, 0.1), predict=False), 4), (dict(stall=(20, 0.5)), 6),
                                        (dict(), 12)])
@pytest.mark.parametrize('k', [1, 3])
def test_no_step_past_a_rule(small, rule, steps, k):  # noqa: F811
    """An operator that GMRES makes no way on (its eigenvalues around the origin): the iteration ends at the rule's step,
    and the preconditioner was applied that many times."""
    geo, ds, od = small
    n = 300
    rng = np.random.default_rng(k)
    A = torch.from_numpy(rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))).to('cuda')
    B = torch.from_numpy(rng.standard_normal((n, k)) + 1j * rng.standard_normal((n, k))).to('cuda')
    calls = []

    def M(R):
        calls.append(1)
        return R.clone()
    Y, it = ds.gmres_batched(lambda V: A @ V, B, M, rtol=1e-10, restart=12 if not rule else 30, **rule)
    assert max(it) == steps and len(calls) == steps
