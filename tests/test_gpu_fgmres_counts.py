"""fgmres with no iterations to take: no cycle runs, and it says so; a right-hand side of
zero needs none."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('kw', [dict(max_iterations=0), dict(max_iterations=-1), dict(max_iterations=0, restart=-1)])
def test_no_iterations(kw):
    import torch
    import dpf_gb300
    b = torch.ones(6, dtype=torch.float64, device='cuda')
    same = lambda v: v
    with pytest.raises(dpf_gb300.SubdivideError, match='did not converge'):
        dpf_gb300.fgmres(same, b, same, **kw)
    x, info = dpf_gb300.fgmres(same, b, same, strict=False, **kw)
    assert not x.any() and info['iterations'] == 0 and info['converged'] is False
    x, info = dpf_gb300.fgmres(same, 0*b, same, **kw)
    assert not x.any() and info == dict(iterations=0, relative_residual=0.)
