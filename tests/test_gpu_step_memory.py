"""The float64 step driver's stored linearisation (46 doubles a bond) is there for the
step alone, and a step that it leaves no memory for runs without it: the allocations
are refused by a stand-in of ``torch.empty``, nothing fills the device."""
import weakref

import pytest

from tests.test_gpu_newton64 import _pair, _same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('refused', [None, 'linearisation', 'tensors beside it'])
def test_linearisation_lives_for_a_step(monkeypatch, refused):
    import torch
    load, python, native = _pair(7, contacts=True)
    size, empty, seen = 46*native.n_bonds, torch.empty, []

    def limited(*shape, **kw):
        if refused == 'linearisation' and shape == ((size,),):
            raise torch.cuda.OutOfMemoryError('refused')
        if refused == 'tensors beside it' and seen and seen[-1]() is not None:
            raise torch.cuda.OutOfMemoryError('refused')
        out = empty(*shape, **kw)
        if out.numel() == size:
            seen.append(weakref.ref(out))
        return out

    for _ in range(2):
        _, ip = python.step(2e-3, python.tensor(load))
        external = native.tensor(load)
        with monkeypatch.context() as patch:
            patch.setattr(torch, 'empty', limited)
            _, inn = native.step(2e-3, external)
        for key in ('nonlinear_iterations', 'krylov_iterations', 'cg_iterations'):
            assert ip[key] == inn[key], key
        assert all(ref() is None for ref in seen)
    assert len(seen) == dict([(None, 2), ('linearisation', 0), ('tensors beside it', 1)])[refused]
    _same(python, native, float(4e-3*python.v.abs().max()))
