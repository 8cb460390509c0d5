"""The Python side of calls that reach the library, with the library's entry points
replaced by a recorder: no GPU is needed, and no address gets further than the recorder."""
import pytest
import torch

from becgpp_b200 import _lib, default_cfg, operators


class _Recorder:
    """Stands for the loaded library: notes every call and reports success."""

    def __init__(self):
        self.calls = []

    def __getattr__(self, name):
        return lambda *a: self.calls.append((name, a)) or 0


@pytest.fixture
def batch(monkeypatch):
    """A HamiltonianBatch of three 16^2 instances without a plan, and the recorder."""
    rec = _Recorder()
    monkeypatch.setattr(_lib, "_lib", rec)
    monkeypatch.setattr(_lib, "stream_ptr", lambda: None)
    monkeypatch.setattr(operators, "_dev_c128", lambda p: p)

    class NoPlan:
        def __init__(self, descs):
            self.handle = None

    monkeypatch.setattr("becgpp_b200.grid.Plan", NoPlan)
    cfgs = [default_cfg(dimension="2D", Ngrid=16, L=6.0, beta2=float(b)) for b in range(3)]
    return operators.HamiltonianBatch(cfgs), rec


def _fields(n, dtype=torch.complex128):
    return [torch.zeros(16, 16, dtype=dtype) for _ in range(n)]


@pytest.mark.parametrize("n", [0, 2, 4])
@pytest.mark.parametrize("which", ["psis", "out", "phis"])
def test_batch_lists_have_one_entry_per_instance(batch, which, n):
    hb, rec = batch
    lists = dict(psis=_fields(3), out=_fields(3), phis=_fields(3, torch.float64))
    lists[which] = lists[which][:n] + _fields(max(0, n - 3))
    with pytest.raises(ValueError):
        hb.apply(lists["psis"], out=lists["out"], phis=lists["phis"])
    assert rec.calls == []                       # nothing was launched


def test_batch_lists_of_the_right_length_reach_the_library(batch):
    hb, rec = batch
    out = _fields(3)
    assert hb.apply(iter(_fields(3)), out=out, phis=_fields(3, torch.float64)) is out
    assert [name for name, _ in rec.calls] == ["bgp_apply_H_batch"]


def test_batch_outputs_own_their_storage(batch):
    hb, _ = batch
    outs = hb.apply(_fields(3))
    for k, o in enumerate(outs):
        o.fill_(k + 1.0)
    assert len({o.untyped_storage().data_ptr() for o in outs}) == 3
    assert [o.untyped_storage().nbytes() for o in outs] == [16 * 16 * 16] * 3
    outs[0].resize_(64, 64).fill_(9.0)           # grows its own storage only
    assert torch.equal(outs[1], torch.full((16, 16), 2.0, dtype=torch.complex128))
    assert torch.equal(outs[2], torch.full((16, 16), 3.0, dtype=torch.complex128))
