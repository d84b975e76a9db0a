"""Row buffers that are moved 16 bytes at a time are refused at other addresses,
before anything is launched (no GPU: the addresses are never followed)."""
import ctypes as C

import pytest


@pytest.fixture(scope="module")
def lib():
    from warp_sph_gpt_gb300 import build

    build.build_cuda()
    from warp_sph_gpt_gb300 import _lib

    return _lib.load()


def _state(off):
    from warp_sph_gpt_gb300 import _lib

    n, g = _lib.MpnnNetT(), _lib.MpnnGradT()
    n.n_nodes, n.n_recv, n.edge_capacity = 4, 2, 8
    at = 1 << 20
    for s in (n, g):
        for name, kind in s._fields_:
            if kind is C.c_void_p:
                setattr(s, name, at + off.get(name, 0))
                at += 1 << 20
    return n, g


@pytest.mark.parametrize("name", ["x", "h0", "agg", "h1", "h2", "h3", "out", "z0", "z2"])
def test_forward_refuses_a_misaligned_row_buffer(lib, name):
    n, _ = _state({name: 8})
    assert lib.sphdem_mpnn_forward(C.byref(n), 1, None) == 2
    assert b"16-byte" in lib.sphdem_last_error()


@pytest.mark.parametrize("name", ["g2", "d_h2", "d_h1", "d_h0", "bf_a", "bf_b"])
def test_backward_refuses_a_misaligned_row_buffer(lib, name):
    n, g = _state({name: 4})
    assert lib.sphdem_mpnn_backward(C.byref(n), C.byref(g), None) == 2
    assert b"16-byte" in lib.sphdem_last_error()
