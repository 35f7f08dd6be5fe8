"""GPU tests of the masked GEMM (matmul_anyway_full_non0tab,
src/impl_matmul_non0tab.rs:163-377) through the C ABI: the reference test's
30 % periodic pattern, masked B entries left NONZERO (the mask alone must
exclude them), transa, ragged blocks, split precision, and the reference's
`unimplemented!` for transb."""
import numpy as np
import pytest

from conftest import check_gemm_summary, load_golden, normwise

pytestmark = pytest.mark.gpu
TOL = 1e-13


def test_matmul_anyway_full_non0tab_golden(cm, wl):
    g = load_golden("matmul_non0tab_pattern30")
    m, n, k, blk = int(g["m"]), int(g["n"]), int(g["k"]), int(g["blksize"])
    a, b, lda, ldb, tab, nblk = wl.ref_matmul_non0tab_inputs(m, n, k, blk)
    c = np.zeros((m, n))
    cm.matmul_anyway_full_non0tab(c, a, b, m, n, k, lda, ldb, n, False, False, tab, nblk)
    check_gemm_summary(c, g, TOL)


@pytest.mark.parametrize("transa", [False, True])
@pytest.mark.parametrize("blk,shape", [(48, (200, 500, 300)), (16, (37, 95, 129)),
                                       (240, (129, 1000, 64))])
def test_non0tab_vs_oracle_nonzero_masked_entries(cm, oracle, transa, blk, shape):
    m, n, k = shape
    rng = np.random.default_rng(m + n + k + blk)
    a = rng.uniform(-1, 1, (k, m) if transa else (m, k))
    b = rng.uniform(-1, 1, (k, n))  # masked entries keep their values
    nblk = -(-n // blk)
    tab = (rng.random((k, nblk)) < 0.3).astype(np.uint8)
    c0 = rng.uniform(-1, 1, (m, n))
    c, ref = c0.copy(), c0.copy()
    cm.MatmulLoops().matmul_loop_parallel_mnk_pack_a_non0tab(c, a, b, m, n, k, a.shape[1], n, n,
                                                             transa, False, tab, nblk, BLKSIZE=blk)
    oracle.matmul_anyway_full_non0tab(ref, a, b, m, n, k, a.shape[1], n, n, transa, False, tab,
                                      nblk, blk)
    assert normwise(c, ref) < TOL


def test_non0tab_any_blksize_vs_dense(cm, wl):
    rng = np.random.default_rng(3)
    m, n, k, blk = 70, 333, 90, 50  # not a multiple of 16: beyond the reference's tiling
    a = rng.uniform(-1, 1, (m, k))
    b = rng.uniform(-1, 1, (k, n))
    nblk = -(-n // blk)
    tab = (rng.random((k, nblk)) < 0.4).astype(np.uint8)
    c = np.zeros((m, n))
    cm.matmul_non0tab_ex(c, a, b, m, n, k, k, n, n, False, False, tab, nblk, blk)
    ref = a @ np.where(wl.expand_mask(tab, n, blk), b, 0.0)
    assert normwise(c, ref) < TOL


def test_non0tab_split_precision(cm, oracle, wl):
    a, b, lda, ldb, tab, nblk = wl.ref_matmul_non0tab_inputs(223, 1000, 223, 48)
    b = b + 0.5  # masked entries nonzero
    c = np.zeros((223, 1000))
    ref = np.zeros((223, 1000))
    cm.matmul_non0tab_ex(c, a, b, 223, 1000, 223, lda, ldb, 1000, False, False, tab, nblk, 48,
                         precision=cm.PREC_OZAKI_INT8)
    oracle.matmul_anyway_full_non0tab(ref, a, b, 223, 1000, 223, lda, ldb, 1000, False, False, tab,
                                      nblk, 48)
    assert normwise(c, ref) < 1e-12


def test_non0tab_transb_is_unimplemented(cm):
    c = np.zeros((4, 48))
    with pytest.raises(NotImplementedError):
        cm.matmul_anyway_full_non0tab(c, np.ones((4, 5)), np.ones((48, 5)), 4, 48, 5, 5, 5, 48,
                                      False, True, np.ones((5, 1), np.uint8), 1)
    assert np.all(c == 0)


def test_non0tab_device_pointers(cm):
    import torch
    m, n, k, blk = 150, 480, 200, 48
    g = torch.Generator(device="cuda").manual_seed(2)
    a = torch.rand(m, k, dtype=torch.float64, device="cuda", generator=g)
    b = torch.rand(k, n, dtype=torch.float64, device="cuda", generator=g)
    tab = (torch.rand(k, n // blk, device="cuda", generator=g) < 0.3).to(torch.uint8)
    c = torch.zeros(m, n, dtype=torch.float64, device="cuda")
    cm.matmul_non0tab_ex(c, a, b, m, n, k, k, n, n, False, False, tab, n // blk, blk)
    torch.cuda.synchronize()
    mask = tab.cpu().numpy().astype(bool).repeat(blk, axis=1)
    ref = a.cpu().numpy() @ np.where(mask, b.cpu().numpy(), 0.0)
    assert normwise(c.cpu().numpy(), ref) < TOL


@pytest.mark.parametrize("prec", [0, 1])
def test_large_masked_host_call_in_blocks(cm, wl, prec):
    """A host-pointer masked GEMM with C above 64 MB runs in blocks of rows
    whose transfers overlap the work: accumulation into a nonzero C, odd
    lda/ldc, the mask whole on the device; (split precision) the same bits as
    one device-pointer call, and within the parity bar of FP64 numpy."""
    import torch
    m, n, k, blk = 1100, 8000, 600, 48
    lda, ldc = k + 5, n + 3
    rng = np.random.default_rng(60 + prec)
    a = rng.uniform(-1, 1, (m, lda))
    b = rng.uniform(-1, 1, (k, n))
    nblk = -(-n // blk)
    tab = (rng.random((k, nblk)) < 0.3).astype(np.uint8)
    c0 = rng.uniform(-1, 1, (m, ldc))
    c = c0.copy()
    cm.matmul_non0tab_ex(c, a, b, m, n, k, lda, n, ldc, False, False, tab, nblk, blk, prec)
    bm = np.where(wl.expand_mask(tab, n, blk), b, 0.0)
    ref = c0[:, :n] + a[:, :k] @ bm
    assert normwise(c[:, :n], ref) < (1e-12 if prec else 1e-13)
    assert np.array_equal(c[:, n:], c0[:, n:])
    if prec:
        dc = torch.from_numpy(c0.copy()).cuda()
        cm.matmul_non0tab_ex(dc, torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda(), m, n, k,
                             lda, n, ldc, False, False, torch.from_numpy(tab).cuda(), nblk, blk,
                             prec)
        torch.cuda.synchronize()
        assert np.array_equal(dc.cpu().numpy(), c)


@pytest.mark.parametrize("transa,m,n,k,blk,density,pad", [
    (False, 128, 256, 65, 32, 0.5, 0),     # one row tile
    (False, 129, 257, 80, 32, 0.6, 0),     # one row past it; odd rows of B are copied
    (True, 130, 130, 90, 64, 0.4, 0),      # A and B in place
    (True, 131, 457, 133, 65, 0.4, 1),     # odd BLKSIZE, two pieces per block
    (False, 40, 1400, 250, 200, 0.2, 2),   # five pieces of 40 columns
    (False, 5, 33, 70, 48, 1.0, 0),        # a block wider than C, every tile present
    (False, 300, 320, 96, 80, 0.0, 0),     # no tile present: C is untouched
    (False, 128, 256, 64, 32, 0.5, 0),     # small: the dense form on zero-filled tiles
    (False, 120, 96, 20000, 48, 0.3, 0),   # lists of more rows than one pass builds
    (False, 1000, 1600, 640, 33, 0.65, 0),  # both forms enqueued, compacted runs
    (False, 1000, 1600, 640, 33, 0.9, 0),  # both forms enqueued, dense runs
])
def test_non0tab_compacted_rows_vs_dense(cm, wl, transa, m, n, k, blk, density, pad):
    """Edges of the compacted form's tiles (128 rows, 16 list rows, pieces of up
    to 64 columns) and its alignment cases; masked entries of B are nonzero, and
    row strides are padded by `pad`.  Empty blocks leave C bit for bit."""
    import torch
    rng = np.random.default_rng(1000 * blk + n)
    a = rng.uniform(-1, 1, (k, m + pad) if transa else (m, k + pad))
    b = rng.uniform(-1, 1, (k, n + pad))
    nblk = -(-n // blk)
    tab = (rng.random((k, nblk)) < density).astype(np.uint8)
    if density < 1.0:
        tab[:, 0] = 0
    if 0.0 < density < 1.0:  # lists of one row, of a full stage of 16, of one more
        for blk_i, rows in zip(range(1, nblk), (1, 16, 17)):
            tab[:, blk_i] = 0
            tab[rng.choice(k, rows, replace=False), blk_i] = 1
    c0 = rng.uniform(-1, 1, (m, n + pad))
    bm = np.where(wl.expand_mask(tab, n, blk), b[:, :n], 0.0)
    ref = c0.copy()
    ref[:, :n] += (a[:, :m].T if transa else a[:, :k]) @ bm
    t = lambda x: torch.from_numpy(x.copy()).cuda()
    c = t(c0)
    cm.matmul_non0tab_ex(c, t(a), t(b), m, n, k, a.shape[1], n + pad, n + pad, transa, False,
                         t(tab), nblk, blk)
    torch.cuda.synchronize()
    c = c.cpu().numpy()
    assert normwise(c, ref) < TOL
    assert np.array_equal(c[:, n:], c0[:, n:])
    if density < 1.0:
        assert np.array_equal(c[:, :min(blk, n)], c0[:, :min(blk, n)])


@pytest.mark.parametrize("transa,m,n,k,blk,density,pad", [
    (False, 260, 1400, 600, 200, 0.2, 0),     # five pieces of 40 columns to a block
    (True, 260, 1450, 600, 145, 0.3, 0),      # odd BLKSIZE: five pieces of 30, B copied
    (True, 457, 1001, 501, 65, 0.4, 1),       # odd sizes and rows throughout
    (False, 129, 3200, 500, 32, 0.5, 0),      # two column pairs to an item; one row past a tile
    (False, 385, 1057, 517, 64, 0.6, 3),      # a last block of 33 columns
    (True, 384, 1056, 518, 48, 0.6, 2),       # A and B in place
    (False, 1500, 33, 5000, 48, 1.0, 0),      # one block, wider than C, all of it present
    (False, 1500, 34, 5000, 2**31 - 1 - 4096, 0.5, 0),  # the widest block there is
    (False, 300, 2400, 300, 80, 0.0, 0),      # no tile present: C is untouched
    (False, 128, 96, 20000, 48, 0.3, 0),      # lists of more rows than one pass builds
    (True, 9, 16384, 1600, 48, 0.4, 1),       # few rows of C
    (False, 1000, 2000, 640, 40, 0.5, 0),     # both forms enqueued, compacted runs
    (False, 1000, 2000, 640, 40, 0.97, 0),    # both forms enqueued, dense runs
    (False, 40, 16384, 1000, 40, 0.2, 0),     # both enqueued for few rows, compacted runs
    (False, 40, 16384, 1000, 40, 0.8, 0),     # and dense
])
def test_non0tab_compacted_form_edges(cm, wl, transa, m, n, k, blk, density, pad):
    """The compacted form (products of more than 4e8 operations, blocks of 32 columns
    and more) at the edges of its tiles and in each of its alignment cases.  Absent
    tiles of B hold NaN, list rows of one, 16 and 17 rows occur, and blocks without a
    present tile leave C bit for bit."""
    import torch
    assert 2.0 * m * n * k > 4e8 and min(blk, n) >= 32
    rng = np.random.default_rng(m + n)
    a = rng.uniform(-1, 1, (k, m + pad) if transa else (m, k + pad))
    b = rng.uniform(-1, 1, (k, n + pad))
    nblk = -(-n // blk)
    tab = (rng.random((k, nblk)) < density).astype(np.uint8)
    if 0.0 < density < 0.9 and nblk > 4:
        tab[:, 0] = 0
        for blk_i, rows in zip(range(1, 4), (1, 16, 17)):
            tab[:, blk_i] = 0
            tab[rng.choice(k, rows, replace=False), blk_i] = 1
    on = np.repeat(tab, min(blk, n), axis=1)[:, :n].astype(bool)
    ref = rng.uniform(-1, 1, (m, n + pad))
    t = lambda x: torch.from_numpy(x.copy()).cuda()
    c0, c = ref.copy(), t(ref)
    ref[:, :n] += (a[:, :m].T if transa else a[:, :k]) @ np.where(on, b[:, :n], 0.0)
    b[:, :n][~on] = np.nan
    cm.matmul_non0tab_ex(c, t(a), t(b), m, n, k, a.shape[1], n + pad, n + pad, transa, False,
                         t(tab), nblk, blk)
    torch.cuda.synchronize()
    c = c.cpu().numpy()
    assert normwise(c, ref) < TOL
    assert np.array_equal(c[:, n:], c0[:, n:])
    empty = ~on.any(axis=0)
    assert np.array_equal(c[:, :n][:, empty], c0[:, :n][:, empty])


def test_non0tab_compacted_form_leaves_out_rows_without_a_present_tile(cm):
    """Row p of op(A)^T meets only the present tiles of row p of B: Inf and NaN there
    do not reach C when there are none (as in the reference's compaction).  The
    zero-filled form of smaller products multiplies them with zeros."""
    import torch
    rng = np.random.default_rng(4)
    m, n, k, blk = 300, 1920, 500, 48
    a, b = rng.uniform(-1, 1, (m, k)), rng.uniform(-1, 1, (k, n))
    tab = (rng.random((k, n // blk)) < 0.3).astype(np.uint8)
    tab[[3, 77, 499]] = 0
    ref = a @ np.where(np.repeat(tab, blk, axis=1).astype(bool), b, 0.0)
    a[:, 3], a[:, 77], a[5, 499] = np.inf, np.nan, -np.inf
    t = lambda x: torch.from_numpy(x).cuda()
    c = torch.zeros(m, n, dtype=torch.float64, device="cuda")
    cm.matmul_non0tab_ex(c, t(a), t(b), m, n, k, k, n, n, False, False, t(tab), n // blk, blk)
    torch.cuda.synchronize()
    assert normwise(c.cpu().numpy(), ref) < TOL


@pytest.mark.parametrize("transa,m,n,k,blk,density,pad", [
    (True, 20000, 62, 500, 4096, 0.5, 0),            # a block wider than C, compacted
    (True, 38000, 64, 200, 2**31 - 1 - 4096, 0.5, 0),  # the widest block there is
    (True, 129, 8000, 1000, 64, 0.3, 1),             # both forms enqueued, compacted runs
    (True, 129, 8000, 1000, 64, 0.95, 1),            # and dense
    (False, 64, 16384, 500, 33, 0.05, 0),            # the dense form alone: few rows, copies
    (True, 9, 16384, 1600, 48, 0.3, 1),              # and where both operands are copied
    (False, 60000, 33, 700, 48, 0.95, 0),            # tall A, one narrow block: dense runs
])
def test_non0tab_forms_by_the_sizes(cm, transa, m, n, k, blk, density, pad):
    """Products that take the compacted form, the dense one or the device's choice by the
    model of both; absent tiles of B hold NaN."""
    import torch
    rng = np.random.default_rng(m + n)
    a = rng.uniform(-1, 1, (k, m + pad) if transa else (m, k + pad))
    b = rng.uniform(-1, 1, (k, n + pad))
    nblk = -(-n // blk)
    tab = (rng.random((k, nblk)) < density).astype(np.uint8)
    on = np.repeat(tab, min(blk, n), axis=1)[:, :n].astype(bool)
    ref = rng.uniform(-1, 1, (m, n + pad))
    t = lambda x: torch.from_numpy(x.copy()).cuda()
    c0, c = ref.copy(), t(ref)
    ref[:, :n] += (a[:, :m].T if transa else a[:, :k]) @ np.where(on, b[:, :n], 0.0)
    b[:, :n][~on] = np.nan
    cm.matmul_non0tab_ex(c, t(a), t(b), m, n, k, a.shape[1], n + pad, n + pad, transa, False,
                         t(tab), nblk, blk)
    torch.cuda.synchronize()
    c = c.cpu().numpy()
    assert normwise(c, ref) < TOL
    assert np.array_equal(c[:, n:], c0[:, n:])
