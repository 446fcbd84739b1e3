"""CPU tests of the alignment checks of the C ABI: an address that does not suit a kernel's vector accesses is refused with a
status, before any CUDA call (the addresses here are never dereferenced)."""
import ctypes

import pytest

from jaxrwkv_b200 import _lib

EUNSUPPORTED = -6
F32, BF16 = _lib.F32, _lib.BF16


def _p(x):
    return ctypes.c_void_p(x)


def _calls(lib, dtype, version=7, residual=True, T=32, flags=0):
    """(name, argument positions of the pointers that are looked at, function of the argument list)."""
    size = 1 << 40
    if version == 7:
        fwd = [_p(4096)] * 9 + [_p(4096), _p(4096), _p(4096) if residual else None, size, flags]
        bwd = [_p(4096)] * 9 + [_p(4096), _p(4096), _p(4096), size] + [_p(4096)] * 7 + [flags]
        return (lambda a: lib.b200wkv7_fwd(None, dtype, 1, T, 1, 64, *a), fwd), (lambda a: lib.b200wkv7_bwd(None, dtype, 1, T, 1, 64, *a), bwd)
    fwd = [_p(4096)] * 8 + [_p(4096), _p(4096), _p(4096) if residual else None, size, flags]
    bwd = [_p(4096)] * 8 + [_p(4096), _p(4096), _p(4096), size] + [_p(4096)] * 6 + [flags]
    return (lambda a: lib.b200wkv6_fwd(None, dtype, version, 1, T, 1, 64, *a), fwd), (lambda a: lib.b200wkv6_bwd(None, dtype, version, 1, T, 1, 64, *a), bwd)


def _refused(call, args, positions, offset):
    for i in positions:
        moved = list(args)
        moved[i] = _p(4096 + offset)
        assert call(moved) == EUNSUPPORTED, (i, offset)


@pytest.mark.parametrize("dtype,flags,least", [(F32, 0, 16), (BF16, _lib.FLAG_SEQUENTIAL, 8), (BF16, 0, 16)])
def test_rwkv7_forward_and_backward(dtype, flags, least):
    (fwd, fa), (bwd, ba) = _calls(_lib.load(), dtype, flags=flags)
    for offset in (2, 4, 8)[:{16: 3, 8: 2}[least]]:
        _refused(fwd, fa, [0, 1, 2, 3, 4, 5, 6, 9, 10], offset)          # streams, s0, y, s_out
        _refused(bwd, ba, [0, 1, 2, 3, 4, 5, 9] + list(range(13, 19)), offset)   # streams, dy, their gradients
    _refused(fwd, fa, [11], 8)                                           # residual
    _refused(bwd, ba, [11], 8)
    _refused(bwd, ba, [6, 10, 19], 4)                                    # s0, ds_out, ds0


@pytest.mark.parametrize("dtype", [F32, BF16])
def test_rwkv7_single_token(dtype):
    (fwd, fa), _ = _calls(_lib.load(), dtype, residual=False, T=1)
    _refused(fwd, fa, [6, 10], 8)
    _refused(fwd, fa, [0, 1, 2, 3, 4, 5], 4)


@pytest.mark.parametrize("dtype,version,least", [(F32, 5, 16), (F32, 6, 16), (BF16, 6, 16), (BF16, 5, 8)])
def test_rwkv6_family(dtype, version, least):
    (fwd, fa), (bwd, ba) = _calls(_lib.load(), dtype, version)
    for offset in (2, 4, 8)[:{16: 3, 8: 2}[least]]:
        _refused(fwd, fa, [0, 1, 2, 3, 8], offset)                       # r k v w, y
        _refused(bwd, ba, [0, 1, 2, 3, 8, 12, 13, 14], offset)           # r k v w, dy, dr dk dv
    _refused(bwd, ba, [9, 17], 4)                                        # ds_out, ds0
    _refused(bwd, ba, [10, 15, 16], 8)                                   # residual, dw, du


@pytest.mark.parametrize("dtype,D,least", [(F32, 64, 16), (BF16, 64, 16), (BF16, 68, 8)])
def test_token_shift(dtype, D, least):
    lib = _lib.load()
    fwd, bwd = [_p(4096)] * 7, [_p(4096)] * 10
    offset = least // 2
    _refused(lambda a: lib.b200wkv_token_shift_fwd(None, dtype, 1, 8, D, 6, *a), fwd, [0, 1, 2, 5, 6], offset)
    _refused(lambda a: lib.b200wkv_token_shift_bwd(None, dtype, 1, 8, D, 6, *a), bwd, [0, 1, 2, 5, 6, 7, 8], offset)
