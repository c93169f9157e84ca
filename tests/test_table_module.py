"""The module that looks over a dict of tensors is tied to the installed torch: it is built anew for another one, and a table
works without it."""
import pytest
import torch

import sharedtensor
from sharedtensor_b200 import _build, _native
from sharedtensor_b200.ops import table


def test_the_module_is_rebuilt_for_another_torch(monkeypatch, tmp_path):
    src = _build.CSRC / "core/tensors.cpp"
    ran = []
    target = tmp_path / "_tensors.so"

    def run(cmd, verbose):
        ran.append(cmd)
        target.touch()

    monkeypatch.setattr(_build, "_run", run)
    monkeypatch.setattr(_build, "OBJ", tmp_path)
    monkeypatch.setattr(_build, "target_path", lambda name: target)
    assert _build.build_tensors() == target and len(ran) == 2, "compiled and linked"
    assert str(src) in ran[0]
    _build.build_tensors()
    assert len(ran) == 2, "built for this torch"
    monkeypatch.setattr(_build, "_torch_version", lambda: "0.0.another")
    _build.build_tensors()
    assert len(ran) == 4
    _build.build_tensors()
    assert len(ran) == 4


def test_a_table_that_cannot_be_made_gives_its_replica_back(free_port, monkeypatch):
    class Broken(table.SharedTable):
        def __init__(self, shared, layout):
            raise MemoryError

    tensors = {"a": torch.zeros(40)}
    monkeypatch.setattr(table, "SharedTable", Broken)
    with pytest.raises(MemoryError):
        sharedtensor.createOrFetchTable("127.0.0.1", free_port, tensors)
    monkeypatch.undo()
    t = sharedtensor.createOrFetchTable("127.0.0.1", free_port, tensors)
    try:
        assert t.shared.is_master, "nobody answers at the port any more"
    finally:
        t.close()


@pytest.mark.gpu
def test_a_table_works_without_the_module(free_port, monkeypatch):
    def missing():
        raise ImportError("undefined symbol")

    monkeypatch.setattr(_native, "tensors", missing)
    init = {"a": torch.randn(40, 30, device="cuda"), "b": torch.randn(7, device="cuda")}
    tab = sharedtensor.createOrFetchTable("127.0.0.1", free_port, init)
    try:
        tab.addFromTensors({k: torch.ones_like(v) for k, v in init.items()})
        out = {k: torch.empty_like(v) for k, v in init.items()}
        tab.copyToTensors(out)
        assert all(torch.equal(out[k], v + 1) for k, v in init.items())
        assert tab.scales()["b"]["sumsq"] == pytest.approx(float(out["b"].double().square().sum()), rel=1e-12)
    finally:
        tab.close()
