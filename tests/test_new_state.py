"""New state tensors come unwritten and are zeroed together: also those of a parameter that is refused half way."""
import pytest
import torch


def _unwritten(monkeypatch):
    """torch.empty as a step may find it: full of what was there before."""
    real = torch.empty

    def empty(*args, **kwargs):
        t = real(*args, **kwargs)
        return t.fill_(113) if t.dtype == torch.uint8 else t.fill_(float("nan"))

    monkeypatch.setattr(torch, "empty", empty)


@pytest.mark.parametrize("dtype,period", [(torch.float64, 4), (torch.float64, 1), (torch.int32, 4)])
def test_codes_of_a_refused_gradient_are_zero(monkeypatch, dtype, period):
    from gefen_b200.gefen import Gefen

    p = torch.nn.Parameter(torch.zeros(24))
    opt = Gefen([p], lr=1e-3)
    state, fresh = opt.state[p], []
    state["automatic_period"] = period
    _unwritten(monkeypatch)
    with pytest.raises(ValueError, match="state dtype is undefined"):
        opt._ensure_state("p", p, p, torch.zeros(24, dtype=dtype), fresh=fresh)
    opt._zeroed(fresh)
    for key in ("m_codebook", "m_magnitude", "vmean"):
        assert key not in state or not bool(state[key].any()), key


@pytest.mark.parametrize("period", [1, 6])
def test_new_state_is_zero(monkeypatch, period):
    from gefen_b200.gefen import Gefen

    p = torch.nn.Parameter(torch.zeros(24))
    opt = Gefen([p], lr=1e-3)
    opt.state[p]["automatic_period"] = period
    fresh = []
    _unwritten(monkeypatch)
    state = opt._ensure_state("p", p, p, torch.zeros(24), fresh=fresh)
    opt._zeroed(fresh)
    assert not any(bool(state[key].any()) for key in ("m_codebook", "m_magnitude", "vmean"))
    assert tuple(state["m_codebook"].shape) == (24 // period, period)
