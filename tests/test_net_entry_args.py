"""The network's entries refuse what would fault on the device, before they touch it: null and misaligned
pointers and rows that are not a multiple of 16 (no GPU needed: every case is refused on the host)."""
import ctypes

import pytest

P = ctypes.c_void_p
BASE = 1 << 20


@pytest.fixture(scope="module")
def lib():
    from lex_gb300 import build, _lib
    build.build()
    return _lib.load()


def arr(n, bad=None, off=0):
    return (P * n)(*[BASE * (i + 1) + (off if i == bad else 0) for i in range(n)])


def forward(lib, nx=16, x=None, w=None, b=None, act=None, pre=None, out=BASE):
    return lib.lexgb_cnn_net_forward(nx, 4, 4, P(x), w or arr(4), b or arr(4), act or arr(4), pre or arr(3), P(out), None)


def backward(lib, nx=16, gout=BASE, w=None, act=None, pre=None, work=BASE, grads=BASE, dx=BASE):
    return lib.lexgb_cnn_net_backward(nx, 4, 4, P(gout), w or arr(4), act or arr(4), pre or arr(3), P(work), P(grads),
                                      P(dx), None)


@pytest.mark.parametrize("off", [2, 4, 8])
@pytest.mark.parametrize("i", range(4))
def test_weights_and_activations_are_16_byte_aligned(lib, i, off):
    from lex_gb300 import _lib
    for call in (forward, backward):
        assert call(lib, w=arr(4, i, off)) == _lib.LEXGB_ERR_ARG
        assert call(lib, act=arr(4, i, off)) == _lib.LEXGB_ERR_ARG
        assert "aligned" in _lib.last_error()
    assert backward(lib, work=BASE + off) == _lib.LEXGB_ERR_ARG


def test_floats_are_4_byte_aligned(lib):
    from lex_gb300 import _lib
    for kw in (dict(x=BASE + 2), dict(out=BASE + 2), dict(b=arr(4, 1, 2)), dict(pre=arr(3, 2, 2)), dict(nx=24)):
        assert forward(lib, **kw) == _lib.LEXGB_ERR_ARG, kw
    for kw in (dict(gout=BASE + 2), dict(grads=BASE + 1), dict(dx=BASE + 2), dict(pre=arr(3, 0, 2)), dict(nx=24)):
        assert backward(lib, **kw) == _lib.LEXGB_ERR_ARG, kw


def test_convolution_operands(lib):
    from lex_gb300 import _lib

    def conv(cin=16, x=BASE, w=BASE, bias=None, pre=None, y=BASE, yf=None):
        return lib.lexgb_cnn_conv3d(16, 4, 4, cin, 32, P(x), P(w), P(bias), P(pre), P(y), P(yf), 1, 32, None)
    for kw in (dict(x=BASE + 8), dict(w=BASE + 4), dict(cin=32, x=BASE + 2), dict(cin=48, x=BASE + 2), dict(y=BASE + 2),
               dict(pre=BASE + 2), dict(yf=BASE + 1), dict(bias=BASE + 2)):
        assert conv(**kw) == _lib.LEXGB_ERR_ARG, kw
