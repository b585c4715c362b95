"""A launch that the runtime refuses is reported by the call that made it and leaves
nothing behind: the caller's next launch does not find its error."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_a_refused_launch_is_reported_once():
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    from seistorch_gb300 import _native, engine
    _native.load(build_if_missing=False)
    dev = torch.device("cuda:0")
    prop = engine.VacousticPropagator(2, 4, 0.001, 10.0, 2, 0, False, dev)
    u = torch.ones(140000, 2, 4, device=dev)  # 70000 pairs: more than a grid's second dimension takes
    with pytest.raises(_native.NativeError):
        prop.kterm(u)
    assert torch.ones(4, device=dev).mul_(2.0).sum().item() == 8.0
    assert prop.kterm(u[:2].contiguous()).shape == (2, 2, 4)
