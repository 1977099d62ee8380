"""Trainer.backward takes as many rows of dL/dY as of X, and no more than the
last forward pass made pre-activations for: anything else is refused before a
kernel is launched (here the library is a recorder on the CPU)."""

import types

import pytest

torch = pytest.importorskip("torch")

from geometricvofext_gb300 import capi, mlp  # noqa: E402


@pytest.fixture
def trainer(monkeypatch):
    launched = []

    class Recorder:
        def __getattr__(self, name):
            return lambda *args: launched.append((name, args)) or 0

    monkeypatch.setattr(capi, "load", lambda *a, **k: Recorder())
    monkeypatch.setattr(mlp.Trainer, "_rows", lambda self, t, dtype: t.to(dtype).contiguous())
    monkeypatch.setattr(torch.cuda, "current_stream", lambda dev=None: types.SimpleNamespace(cuda_stream=0))
    return mlp.Trainer(*mlp.init_params(1), 256, device="cpu"), launched


def _rows(n, dtype=torch.bfloat16):
    return torch.zeros((n, mlp.WIDTH), dtype=dtype)


@pytest.mark.parametrize("fwd,x,dy", [(256, 256, 128), (256, 128, 256), (128, 256, 256), (0, 128, 128)])
def test_row_counts_that_do_not_match_are_refused(trainer, fwd, x, dy):
    tr, launched = trainer
    if fwd:
        tr.forward(_rows(fwd))
    del launched[:]
    with pytest.raises(RuntimeError, match="rows"):
        tr.backward(_rows(x), _rows(dy, torch.float32))
    assert launched == []


@pytest.mark.parametrize("fwd,x", [(256, 256), (192, 192), (256, 128)])
def test_matching_row_counts_are_taken(trainer, fwd, x):
    tr, launched = trainer
    tr.forward(_rows(fwd))
    tr.backward(_rows(x), _rows(x, torch.float32))
    assert [(name, a[2] if name.endswith("backward") else a[1]) for name, a in launched] == [
        ("simplic_mlp_train_forward", fwd), ("simplic_mlp_train_backward", x)]
