"""GPU tests of the host calls on pageable arrays large enough to go through the
library's own pinned buffers: only the present tiles of phi go up (masked entries
hold NaN here, and a first call with every tile present leaves other values on the
device), ragged last tiles, and products whose operands and C go up and come back
in pieces."""
import numpy as np
import pytest

from conftest import normwise

pytestmark = pytest.mark.gpu


def _table(rng, wl, nao, ngrid, blk, density):
    nblk = -(-ngrid // blk)
    tab = (rng.random((nao, nblk)) < density).astype(np.uint8)
    ao = rng.standard_normal((nao, ngrid))
    on = wl.expand_mask(tab, ngrid, blk)
    return np.where(on, ao, np.nan), np.where(on, ao, 0.0), tab


@pytest.mark.parametrize("prec,nao,ngrid,blk,density,two", [
    (0, 301, 4001, 48, 0.3, False),   # odd rows, a last tile of 17 points
    (0, 300, 8192, 64, 0.05, True),   # two tables, rows of few tiles
    (1, 260, 5000, 100, 0.4, True),   # split precision, row form
    (1, 1100, 8230, 64, 0.3, False),  # split precision, pair form
])
def test_only_present_tiles_go_up(cm, wl, prec, nao, ngrid, blk, density, two):
    import torch
    rng = np.random.default_rng(nao + blk)
    d = rng.standard_normal((2, nao, nao))
    full = rng.standard_normal((nao, ngrid))
    ones = np.ones((nao, -(-ngrid // blk)), np.uint8)
    rho = np.zeros((2, ngrid))
    strides = shape = (nao, ngrid)
    cm.aodmao2rho_ex(rho, d, full, full, strides, shape, 2, ones, ones.shape[1], blk, prec)
    lhs, lhs0, tab = _table(rng, wl, nao, ngrid, blk, density)
    rhs, rhs0 = lhs, lhs0
    if two:
        rhs0 = np.where(wl.expand_mask(tab, ngrid, blk), rng.standard_normal((nao, ngrid)), 0.0)
        rhs = np.where(wl.expand_mask(tab, ngrid, blk), rhs0, np.nan)
    rho = np.zeros((2, ngrid))
    cm.aodmao2rho_ex(rho, d, lhs, rhs, strides, shape, 2, tab, tab.shape[1], blk, prec)
    t = lambda x: torch.from_numpy(x).cuda()
    dl = t(lhs0)
    want = torch.zeros(2, ngrid, dtype=torch.float64, device="cuda")
    cm.aodmao2rho_ex(want, t(d), dl, t(rhs0) if two else dl, strides, shape, 2, t(tab),
                     tab.shape[1], blk, prec)
    torch.cuda.synchronize()
    assert np.array_equal(rho, want.cpu().numpy())


def test_fock_present_tiles_go_up(cm, wl):
    rng = np.random.default_rng(3)
    nao, ngrid, blk = 400, 4001, 48
    ao, ao0, tab = _table(rng, wl, nao, ngrid, blk, 0.3)
    w = rng.standard_normal((1, ngrid))
    v = np.zeros((1, nao, nao))
    cm.aodm_fock(v, w, ao, ao, (nao, ngrid), (nao, ngrid), 1, tab, tab.shape[1], blk)
    on = wl.expand_mask(tab, ngrid, blk)
    assert normwise(v[0], (ao0 * w[0]) @ ao0.T) < 1e-13
    assert on.any()


@pytest.mark.parametrize("prec,transa,m,n,k,pad", [
    (0, False, 700, 801, 600, 0),     # pieces of a few rows each
    (0, True, 333, 2000, 1501, 3),
    (1, False, 1500, 6000, 300, 1),   # C above 64 MB: blocks of rows, 2-D pieces
    (0, False, 1500, 6000, 300, 1),   # and of columns
])
def test_products_of_pageable_arrays(cm, prec, transa, m, n, k, pad):
    rng = np.random.default_rng(m)
    a = rng.uniform(-1, 1, (k, m + pad) if transa else (m, k + pad))
    b = rng.uniform(-1, 1, (k, n + pad))
    c0 = rng.uniform(-1, 1, (m, n + pad))
    c = c0.copy()
    cm.matmul_ex(c, a, b, m, n, k, a.shape[1], n + pad, n + pad, transa, False, prec)
    ref = c0[:, :n] + (a[:, :m].T if transa else a[:, :k]) @ b[:, :n]
    assert normwise(c[:, :n], ref) < (1e-12 if prec else 1e-13)
    assert np.array_equal(c[:, n:], c0[:, n:])


def test_buffers_are_given_back_and_made_again(cm):
    rng = np.random.default_rng(8)
    a, b = rng.uniform(-1, 1, (500, 400)), rng.uniform(-1, 1, (400, 600))
    for _ in range(2):
        c = np.zeros((500, 600))
        cm.matmul_anyway_full(c, a, b, 500, 600, 400, 400, 600, 600, False, False)
        assert normwise(c, a @ b) < 1e-13
        cm._raise(cm.lib().cfgmm_release_workspace())


def test_two_threads_at_once(cm):
    import threading
    rng = np.random.default_rng(9)
    jobs = [(rng.uniform(-1, 1, (400 + 50 * i, 500)), rng.uniform(-1, 1, (500, 700)))
            for i in range(4)]
    out = [None] * 4

    def go(i):
        a, b = jobs[i]
        c = np.zeros((a.shape[0], 700))
        cm.matmul_anyway_full(c, a, b, a.shape[0], 700, 500, 500, 700, 700, False, False)
        out[i] = c

    ts = [threading.Thread(target=go, args=(i,)) for i in range(4)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for (a, b), c in zip(jobs, out):
        assert normwise(c, a @ b) < 1e-13


@pytest.mark.parametrize("m,n,k", [
    (128, 6000, 1050),  # A just past 1 MB, B past 48 MB, C of a few MB
    (2000, 64, 1100),   # A past 16 MB, B by the driver
    (131, 137, 1000),   # A just short of 1 MB
])
def test_products_on_either_side_of_the_upload_rules(cm, m, n, k):
    rng = np.random.default_rng(m + n)
    a, b, c0 = rng.uniform(-1, 1, (m, k)), rng.uniform(-1, 1, (k, n)), rng.uniform(-1, 1, (m, n))
    c = c0.copy()
    cm.matmul_ex(c, a, b, m, n, k, k, n, n, False, False)
    assert normwise(c, c0 + a @ b) < 1e-13
