"""The C description of a matrix that the hot calls keep (DenseQ._described), with stand-ins for the library and for device
tensors: what it says, how long it lives and when it is built again."""
import copy
import pickle
import types

import pytest
import torch

from ingot_b200 import capi, linear
from ingot_b200.linear import DenseQ, VQMV


def bare_matrix(N=16, K=64):
    m = DenseQ.__new__(DenseQ)  # (the constructor refuses CPU tensors)
    m.had, m._rot = None, None
    m.w, m.s, m.b = torch.zeros(N, K // 8, dtype=torch.int32), torch.zeros(N, 1, dtype=torch.bfloat16), torch.zeros(N, 1, dtype=torch.bfloat16)
    m.N, m.K, m.bits, m.gs, m.mode, m.experts = N, K, 4, 64, "affine", 1
    return m


def rows(n, k, dtype=torch.float32):
    t = torch.zeros(n, k, dtype=dtype)
    return types.SimpleNamespace(is_cuda=True, dtype=dtype, dim=t.dim, stride=t.stride, data_ptr=t.data_ptr, keep=t)


@pytest.fixture
def fake(monkeypatch):
    """capi with a context and calls that record what they are given."""
    f = types.SimpleNamespace(seen=[], contexts=[], during=lambda: None)

    def qmv(ctx, stream, x, xd, ldx, q, *rest):
        f.during()
        d = capi.QLinear.from_address(q)
        f.contexts.append(ctx)
        f.seen.append((d.w, d.scales, d.biases, d.n, d.k))
        return 0

    monkeypatch.setattr(capi, "context", lambda device=0: types.SimpleNamespace(address=device + 1, check=lambda st: None, device=device, handle=None))
    monkeypatch.setattr(capi, "call", lambda: types.SimpleNamespace(qmv=qmv))
    return f


def encode(m):
    VQMV.encode(rows(1, m.K), m, rows(1, m.N), 1, stream=types.SimpleNamespace(cuda_stream=0))


def test_description_outlives_an_assignment_during_the_call(fake, monkeypatch):
    """Another thread may assign to the matrix while a launch runs without the interpreter lock: what the call reads stays."""
    freed = []

    class Tracked(capi.QLinear):
        def __del__(self):
            freed.append(True)

    monkeypatch.setattr(linear.capi, "QLinear", Tracked)
    m = bare_matrix()
    w0 = m.w

    def during():
        m.w = torch.ones_like(w0)
        assert not freed

    fake.during = during
    encode(m)
    assert fake.seen[0][0] == w0.data_ptr()


def test_description_is_whole_for_a_second_thread(fake):
    """A thread that finds the cached description finds its address too: the second thread is let in wherever the first one
    stores something."""
    inner = []

    class Interleaved(DenseQ):
        def __setattr__(self, name, value):
            super().__setattr__(name, value)
            if name == "_ql" and value is not None:
                encode(self)
                inner.append(fake.seen[-1])

    m = bare_matrix()
    m.__class__ = Interleaved
    encode(m)
    want = (m.w.data_ptr(), m.s.data_ptr(), m.b.data_ptr(), m.N, m.K)
    assert inner == [want] and fake.seen[-1] == want


def test_description_follows_assignments(fake):
    m = bare_matrix()
    encode(m)
    first = m._described()
    assert m._described() is first  # built once
    m.w, m.N = torch.zeros(32, 8, dtype=torch.int32), 32
    m.s, m.b = torch.zeros(32, 1, dtype=torch.bfloat16), torch.zeros(32, 1, dtype=torch.bfloat16)
    encode(m)
    assert fake.seen[-1] == (m.w.data_ptr(), m.s.data_ptr(), m.b.data_ptr(), 32, 64)


@pytest.mark.parametrize("name", ["w", "s", "b"])
def test_description_follows_an_exchanged_storage(fake, name):
    """t.data = ... exchanges the memory under a tensor without an assignment to the matrix."""
    m = bare_matrix()
    encode(m)
    getattr(m, name).data = torch.ones_like(getattr(m, name))
    encode(m)
    assert fake.seen[-1] == (m.w.data_ptr(), m.s.data_ptr(), m.b.data_ptr(), m.N, m.K)


def test_a_used_matrix_copies_and_pickles(fake):
    m = bare_matrix()
    encode(m)
    for c in (copy.copy(m), copy.deepcopy(m), pickle.loads(pickle.dumps(m))):
        encode(c)
        assert fake.seen[-1] == (c.w.data_ptr(), c.s.data_ptr(), c.b.data_ptr(), m.N, m.K)
    assert copy.deepcopy(m).w.data_ptr() != m.w.data_ptr()


def test_context_follows_the_matrix_to_another_device(fake, monkeypatch):
    """A matrix whose codes are assigned from another GPU is launched with that GPU's context."""
    m = bare_matrix()
    where = [0]
    monkeypatch.setattr(DenseQ, "device_index", property(lambda self: where[0]))
    encode(m)
    where[0], m.w = 1, m.w.clone()
    encode(m)
    assert fake.contexts == [1, 2]


def test_ffn_scratch_follows_the_matrices(fake, monkeypatch):
    """The scratch of a dense FFN is sized for the widths its matrices have at the call, also when their fields were assigned."""
    def bytes_of(ctx, gu, dn, rows, x_dtype, n):
        n._obj.value = 1000 * rows * dn._obj.k
        return 0

    given = []
    monkeypatch.setattr(capi, "lib", lambda: types.SimpleNamespace(iq_dense_ffn_workspace_bytes=bytes_of))
    monkeypatch.setattr(capi, "call", lambda: types.SimpleNamespace(dense_ffn=lambda *a: given.append(a[15]) or 0))
    mlp = linear.DenseMLP(bare_matrix(128, 64), bare_matrix(64, 64))
    step = lambda: mlp.encode(rows(2, 64), rows(2, 64), 2, stream=types.SimpleNamespace(cuda_stream=0))
    step()
    step()
    for m, n, k in ((mlp.gate_up, 256, 64), (mlp.down, 64, 128)):
        m.w, m.N, m.K = torch.zeros(n, k // 8, dtype=torch.int32), n, k
    step()
    assert given == [1000 * 2 * 64] * 2 + [1000 * 2 * 128]
