"""The calls on host arrays (ep_align, ep_embed_features) whose result shares
memory with an input, is larger than one download slab, or is refused for one
bad id among many: the result is that of a call on separate arrays, and a
refused call leaves its result array alone."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from cloverleaf_gb300 import _native

pytestmark = pytest.mark.gpu
MB = 1 << 20
INVALID_ARG = -1         # EP_ERR_INVALID_ARG


def _graph(n, deg, seed):
    rng = np.random.default_rng(seed)
    rows = np.arange(n + 1, dtype=np.uint64) * deg
    cols = rng.integers(0, n, n * deg).astype(np.uint32)
    cdf = np.tile((np.arange(deg) + 1) / deg, n).astype(np.float32)
    return rows, cols, cdf


def _align(rows, cols, cdf, dims, emb, alpha, out):
    return _native.lib().ep_align(0, len(rows) - 1, _native.ptr(rows), _native.ptr(cols), _native.ptr(cdf), dims,
                                  ctypes.c_void_p(emb), alpha, 0, ctypes.c_void_p(out))


def _buffer(nbytes, pinned):
    """(keep-alive, address) of nbytes of host memory."""
    if pinned:
        t = torch.empty(nbytes, dtype=torch.uint8, pin_memory=True)
        return t, t.data_ptr()
    a = np.empty(nbytes, np.uint8)
    return a, a.ctypes.data


def _view(addr, shape):
    return np.ctypeslib.as_array(ctypes.cast(addr, ctypes.POINTER(ctypes.c_float)), shape)


@pytest.mark.parametrize("pinned", [False, True])
@pytest.mark.parametrize("mb", [20, 64])
def test_alignment_in_place(mb, pinned):
    dims = 128
    n = mb * MB // (4 * dims)
    rows, cols, cdf = _graph(n, 4, mb)
    emb = np.random.default_rng(mb).standard_normal((n, dims)).astype(np.float32)
    want = _native.align(rows, cols, cdf, emb, alpha=0.25)
    keep, at = _buffer(emb.nbytes, pinned)
    both = _view(at, (n, dims))
    both[:] = emb
    assert _align(rows, cols, cdf, dims, at, 0.25, at) == _native.EP_OK
    assert np.array_equal(both, want)


@pytest.mark.parametrize("pinned", [False, True])
def test_embeddings_over_their_table(pinned):
    # the result begins inside the feature table and is four times as large
    n, dims, n_feat = 140_000, 128, 35_000
    rng = np.random.default_rng(7)
    fptr = np.arange(n + 1, dtype=np.uint64) * 3
    fids = rng.integers(0, n_feat, 3 * n).astype(np.uint32)
    table = rng.standard_normal((n_feat, dims)).astype(np.float32)
    want = _native.embed_features(fptr, fids, table)
    keep, at = _buffer(table.nbytes + want.nbytes, pinned)
    _view(at, table.shape)[:] = table
    out = at + table.nbytes // 2
    assert _native.lib().ep_embed_features(0, n, _native.ptr(fptr), _native.ptr(fids), None, n_feat, dims,
                                           ctypes.c_void_p(at), ctypes.c_void_p(out)) == _native.EP_OK
    assert np.array_equal(_view(out, want.shape), want)


@pytest.mark.parametrize("dims,offset", [(128, 0), (126, 4), (128, 12)])
def test_results_of_several_slabs(oracle, dims, offset):
    # several slabs and a ragged last one, at odd addresses
    n = 72 * MB // (4 * dims) + 1
    rows, cols, cdf = _graph(n, 3, dims)
    emb = np.random.default_rng(dims).standard_normal((n, dims)).astype(np.float32)
    want = oracle.align(rows, cols, cdf, emb, alpha=0.5)
    buf = np.full(want.nbytes + offset + 64, 0xa5, np.uint8)
    out = buf.ctypes.data + offset
    assert _align(rows, cols, cdf, dims, emb.ctypes.data, 0.5, out) == _native.EP_OK
    assert np.array_equal(_view(out, want.shape), want)
    assert (buf[:offset] == 0xa5).all() and (buf[offset + want.nbytes:] == 0xa5).all()


@pytest.mark.parametrize("ids", [131_072, 131_076, 900_000])
def test_one_bad_id_is_refused(oracle, ids):
    # up to 131,072 ids are checked by the host, more by the device
    n, dims = ids // 4, 16
    rows, cols, cdf = _graph(n, 4, ids)
    emb = np.random.default_rng(3).standard_normal((n, dims)).astype(np.float32)
    fptr = rows
    good = _native.align(rows, cols, cdf, emb, alpha=0.5)
    assert np.array_equal(good, oracle.align(rows, cols, cdf, emb, alpha=0.5))
    means = _native.embed_features(fptr, cols, emb)
    assert np.allclose(means, emb[cols].reshape(n, 4, dims).mean(1), rtol=0, atol=1e-5)
    for where in (0, ids - 1):
        bad = cols.copy()
        bad[where] = n
        out = np.full((n, dims), 7.0, np.float32)
        assert _align(rows, bad, cdf, dims, emb.ctypes.data, 0.5, out.ctypes.data) == INVALID_ARG
        assert _native.lib().ep_embed_features(0, n, _native.ptr(fptr), _native.ptr(bad), None, n, dims, _native.ptr(emb),
                                               _native.ptr(out)) == INVALID_ARG
        assert (out == 7.0).all()
