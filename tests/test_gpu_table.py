"""The kernels over a table of tensors against PyTorch."""
import math
import threading
import time

import pytest
import torch

import sharedtensor
from sharedtensor_b200 import _native

pytestmark = pytest.mark.gpu


def _table(sizes, offset=0, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return {f"t{i}": torch.randn(n + offset, generator=g, device="cuda")[offset:] * 2.0 ** -(i % 7) for i, n in enumerate(sizes)}


@pytest.mark.parametrize("sizes,offset", [
    ([1], 0), ([3, 1, 5], 1), ([4095, 4096, 4097, 31, 33], 0), ([4097, 8192], 3), ([16384 * 3 + 5, 2, 16384], 0),
    ([7] * 300, 0), ([100_003, 1, 2_000_001], 2)])
def test_table_of_tensors(free_port, sizes, offset):
    """One tensor, tensors around the chunk sizes, misaligned ones, and more tensors than one launch takes."""
    init = _table(sizes)
    tab = sharedtensor.createOrFetchTable("127.0.0.1", free_port, init)
    try:
        deltas = _table(sizes, seed=1)
        store = {k: torch.zeros(v.numel() + offset, device="cuda") for k, v in init.items()}
        out = {k: v[offset:] for k, v in store.items()}
        for _ in range(2):
            tab.addFromTensors({k: torch.cat([torch.zeros(offset, device="cuda"), v])[offset:] for k, v in deltas.items()})
            tab.copyToTensors(out)
        for k in init:
            assert torch.equal(out[k], (init[k] + deltas[k]) + deltas[k]), k
            assert not store[k][:offset].any()
        flat = tab.copyToFlat(tab.new_flat())
        assert float(flat.double().abs().sum()) == pytest.approx(sum(float(v.double().abs().sum()) for v in out.values()), rel=1e-12)
        for got in (tab.scales(), tab.scales(flat)):
            for k, v in out.items():
                sumsq = float(v.double().square().sum())
                padded = (v.numel() + 31) // 32 * 32
                assert got[k]["sumsq"] == pytest.approx(sumsq, rel=1e-12), k
                assert got[k]["rms_exp"] == math.floor(math.log2(math.sqrt(sumsq / padded))), k
    finally:
        tab.close()


def test_table_tensors_that_need_a_conversion(free_port):
    init = {"a": torch.randn(40, 30, device="cuda"), "b": torch.randn(7, device="cuda")}
    tab = sharedtensor.createOrFetchTable("127.0.0.1", free_port, init)
    try:
        tab.addFromTensors({"a": torch.ones(30, 40, device="cuda").t(), "b": torch.ones(7, dtype=torch.float64)})
        out = {"a": torch.empty(30, 40, device="cuda").t(), "b": torch.empty(7, dtype=torch.bfloat16, device="cuda")}
        tab.copyToTensors(out)
        assert torch.equal(out["a"], init["a"] + 1) and torch.equal(out["b"], (init["b"] + 1).to(torch.bfloat16))
        with pytest.raises(RuntimeError):
            tab.addFromTensors({"a": torch.ones(3, device="cuda"), "b": torch.ones(7, device="cuda")})
    finally:
        tab.close()


def test_names_that_share_memory_are_filled_one_after_the_other(free_port):
    """The later name wins where two overlap, as it does when they are copied in turn."""
    n = 300_000
    init = {"a": torch.randn(n, device="cuda"), "b": torch.randn(n, device="cuda"), "none": torch.empty(0, device="cuda")}
    tab = sharedtensor.createOrFetchTable("127.0.0.1", free_port, init)
    try:
        for shift in (0, 1, n // 2, n - 1, n):
            store = torch.zeros(2 * n, device="cuda")
            want = store.clone()
            want[:n] = init["a"]
            want[shift:shift + n] = init["b"]
            for _ in range(5):
                store.zero_()
                tab.copyToTensors({"a": store[:n], "b": store[shift:shift + n], "none": torch.empty(0, device="cuda")})
                assert torch.equal(store, want), shift
            # (what is read may overlap as it likes)
            tab.addFromTensors({"a": store[:n], "b": store[shift:shift + n], "none": torch.empty(0, device="cuda")})
            init["a"] += store[:n]
            init["b"] += store[shift:shift + n]
    finally:
        tab.close()


def test_tensors_without_memory(free_port):
    """Zeros that are not stored anywhere are added like any others; nothing is read from where a storage used to be."""
    init = {"a": torch.randn(40, 30, device="cuda"), "b": torch.randn(7, device="cuda")}
    tab = sharedtensor.createOrFetchTable("127.0.0.1", free_port, init)
    try:
        tab.addFromTensors({"a": torch._efficientzerotensor((40, 30), device="cuda"), "b": torch.ones(7, device="cuda")})
        out = {k: torch.empty_like(v) for k, v in init.items()}
        tab.copyToTensors(out)
        assert torch.equal(out["a"], init["a"]) and torch.equal(out["b"], init["b"] + 1)
        gone = torch.ones(40, 30, device="cuda")
        gone.untyped_storage().resize_(0)
        assert tab._addresses({"a": gone, "b": out["b"]}, False) is None
        assert tab._addresses(out, False) is not None
    finally:
        tab.close()


def test_layouts_of_a_callers_own(free_port):
    """Tensors without padding between them, and a layout that is not the shared tensor's size."""
    from sharedtensor_b200.ops.table import SharedTable, TableLayout

    shapes = {"a": torch.Size([5]), "b": torch.Size([4097]), "c": torch.Size([2, 3])}
    lay = TableLayout(shapes, 1)
    init = torch.randn(lay.numel, device="cuda")
    st = sharedtensor.createOrFetch("127.0.0.1", free_port, init)
    try:
        tab = SharedTable(st, lay)
        deltas = {k: torch.randn(v, device="cuda") for k, v in shapes.items()}
        tab.addFromTensors(deltas)
        out = {k: torch.empty(v, device="cuda") for k, v in shapes.items()}
        tab.copyToTensors(out)
        for k, v in lay.views(init).items():
            assert torch.equal(out[k], v + deltas[k])
        got = tab.scales()
        for k, v in out.items():
            assert got[k]["sumsq"] == pytest.approx(float(v.double().square().sum()), rel=1e-12)
        other = SharedTable(st, TableLayout({"a": torch.Size([lay.numel + 1])}, 32))
        for call in (other.addFromTensors, other.copyToTensors):
            with pytest.raises(ValueError):
                call({"a": torch.zeros(lay.numel + 1, device="cuda")})
    finally:
        st.close()


def test_every_push_reaches_the_other_replica(free_port):
    """The push sets the change marks of the arena tiles it touches itself: more tensors than one launch takes, tensors that
    straddle tiles, the last of them within one chunk; all of them changed, then one at a time."""
    sizes = [7] * 280 + [5000, 3 * 4096 + 5, 1, 9000, 3000]
    init = _table(sizes)
    a = sharedtensor.createOrFetchTable("127.0.0.1", free_port, init, rejoin=False)
    b = sharedtensor.createOrFetchTable("127.0.0.1", free_port, {k: torch.zeros_like(v) for k, v in init.items()}, rejoin=False)
    try:
        names = list(init)
        expect = {k: v.clone() for k, v in init.items()}
        out = {k: torch.empty_like(v) for k, v in init.items()}
        deltas = {k: torch.zeros_like(v) for k, v in init.items()}
        assert a.flush(10.0) and b.flush(10.0)   # the marks of a new edge are gone
        for changed in (names, [names[0]], [names[255]], [names[256]], *([k] for k in names[-5:])):
            for k in names:
                deltas[k].zero_()
            for k in changed:
                deltas[k].copy_(torch.randn_like(deltas[k]))
                expect[k] += deltas[k]
            a.addFromTensors(deltas)
            assert a.flush(10.0) and b.flush(10.0)
            b.copyToTensors(out)
            for k in changed:
                assert ((out[k] - expect[k]).norm() / expect[k].norm()).item() < 1e-5, (k, len(changed))
    finally:
        b.close()
        a.close()


def test_magnitudes_go_by_the_names_of_the_call(free_port):
    """Another thread may change the names while the call waits for its turn, and any sequence of names will do."""
    init = _table([100, 5000, 3])
    tab = sharedtensor.createOrFetchTable("127.0.0.1", free_port, init)
    try:
        want, got = tab.scales(), []
        busy = torch.cuda.Stream()

        def read_behind(ns):
            with torch.cuda.stream(busy):
                if ns:
                    _native.cuda().delay(ns, busy.cuda_stream)
                got.append(tab.scales())

        threads = [threading.Thread(target=read_behind, args=(ns,)) for ns in (1_000_000_000, 0)]
        for t in threads:
            t.start()
            time.sleep(0.2)
        tab.layout.names[0] = "another"
        for t in threads:
            t.join()
        assert got == [want, want]
        tab.layout.names = tuple(init)
        assert tab.scales() == want
        tab.layout.names = list(init)[:2]
        assert tab.scales() == {k: want[k] for k in list(init)[:2]}
    finally:
        tab.close()
