"""Rounds publish at device scope where every ring stays on this GPU and in this process, at system scope otherwise."""
import multiprocessing as mp
import os
import socket

import pytest
import torch

import sharedtensor
import test_gpu_round_kinds as kinds
from sharedtensor_b200 import _native
from sharedtensor_b200.parallel.local_wiring import connect_local


def connect_undeclared(a, b):
    """An edge of which nothing is said about where its far end lives, as one to another GPU."""
    (la, ba), (lb, bb) = [(r.add_link(), r.alloc_edge_block()) for r in (a, b)]
    return a.attach_peer(la, ba, b.edge_block_ptr(bb)), b.attach_peer(lb, bb, a.edge_block_ptr(ba))


@pytest.fixture
def system_scope(monkeypatch):
    """Edges of which nothing is said about where their far end lives."""
    attach = _native.cuda().GpuReplica.attach_peer
    monkeypatch.setattr(_native.cuda().GpuReplica, "attach_peer", lambda r, link, block, remote, same_gpu=False: attach(r, link, block, remote))
    a, b = [_native.cuda().GpuReplica(0, 5000, _native.cuda().GpuConfig()) for _ in range(2)]
    connect_local(a, b)
    assert not a.one_gpu() and not b.one_gpu()


@pytest.mark.gpu
@pytest.mark.parametrize("bits,block", [(1, 256), (1, 4096), (2, 1024), (4, 32), (8, 32), (8, 4096)])
@pytest.mark.parametrize("topology,members", [("mesh", 3), ("mesh", 8), ("star", 4)])
def test_group_bit_exact_at_system_scope(system_scope, topology, members, bits, block):
    """Members, an inner node and its leaves, in every format, as they are between processes and GPUs."""
    kinds.test_round_bit_exact_in_a_group(topology, members, bits, block)


@pytest.mark.gpu
@pytest.mark.parametrize("topology,members", [("mesh", 2), ("mesh", 4), ("star", 4)])
def test_many_tiles_per_group_at_system_scope(system_scope, topology, members):
    """Half a bank of descriptors is published before the pass has ended."""
    kinds.test_round_bit_exact_with_many_tiles_per_group(topology, members)


@pytest.mark.gpu
@pytest.mark.parametrize("bits,block", [(1, 1024), (8, 32), (8, 4096)])
@pytest.mark.parametrize("topology,members", [("mesh", 2), ("mesh", 4), ("star", 4)])
def test_a_wait_that_runs_out_at_system_scope(system_scope, topology, members, bits, block):
    kinds.test_a_wait_that_runs_out_leaves_no_visit_half_done(topology, members, bits, block, 3)


@pytest.mark.gpu
@pytest.mark.parametrize("members", [2, 4])
def test_round_bit_exact_at_system_scope(monkeypatch, members):
    """(Device scope is what the tests of the kinds of round use.)"""
    torch.manual_seed(members)
    monkeypatch.setattr(kinds, "connect_local", connect_undeclared)
    g = kinds.Group("star", members, 40 * 4096 + 7, 8, 32)
    assert not any(r.one_gpu() for r in g.reps)
    for i in range(members):
        g.add(i, torch.randn(g.n))
    for it in range(4):
        for i in range(members):
            g.visit(i)
            g.check(i, f"in pass {it}")
    g.done()


@pytest.mark.gpu
def test_one_ring_decides():
    cu = _native.cuda()
    a, b, c = [cu.GpuReplica(0, 5000, cu.GpuConfig()) for _ in range(3)]
    connect_local(a, b)
    assert a.one_gpu() and b.one_gpu()
    peer, _ = connect_undeclared(a, c)
    assert not a.one_gpu() and b.one_gpu() and not c.one_gpu()
    a.detach_peer(peer)
    assert a.one_gpu()


@pytest.mark.gpu
def test_two_replicas_of_one_process(free_port):
    x = torch.zeros(1000, device="cuda")
    with sharedtensor.createOrFetch("127.0.0.1", free_port, x) as a, sharedtensor.createOrFetch("127.0.0.1", free_port, x) as b:
        assert a._b.rep.one_gpu() and b._b.rep.one_gpu()


def test_whether_the_other_end_of_a_socket_is_in_this_process():
    cu = _native.cuda()
    name = f"\0sharedtensor-test-{os.getpid()}"
    with socket.socket(socket.AF_UNIX) as server:
        server.bind(name)
        server.listen(2)
        with socket.socket(socket.AF_UNIX) as here:
            here.connect(name)
            conn, _ = server.accept()
            with conn:
                assert cu.unix_same_process(here.fileno()) and cu.unix_same_process(conn.fileno())
        child = mp.get_context("spawn").Process(target=_connect_and_wait, args=(name,))
        child.start()
        try:
            server.settimeout(60)  # (a child that fails never comes)
            conn, _ = server.accept()
            with conn:
                assert not cu.unix_same_process(conn.fileno())
                conn.send(b"x")
            child.join(60)
            assert child.exitcode == 0
        finally:
            child.kill()  # (does nothing to one that has ended)
            child.join()
    assert not cu.unix_same_process(-1)


def _connect_and_wait(name):
    with socket.socket(socket.AF_UNIX) as s:
        s.connect(name)
        s.recv(1)
