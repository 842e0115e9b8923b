"""Products at the sizes where the specialised kernels change over: edges of tiles, remainders, smallest and largest of
their ranges. Checked against the dense product of the decompressed block, relative to the summed magnitudes."""
import numpy as np
import pytest

from systemds_b200 import CompressedMatrixBlock, datagen
from systemds_b200 import colgroup as cg
from systemds_b200.cmb import CHAIN_XtwXv, CLALibDecompress, CLALibLeftMultBy, CLALibMMChain, CLALibRightMultBy, CLALibTSMM
from systemds_b200.mapping import MapToFactory
from systemds_b200.offset import OffsetFactory
from tests.util import TOL, abs_dense_of, dense_of, rel_err

pytestmark = pytest.mark.gpu


def _ddc(nRows, cards, seed, const=False, width=1):
    rng = np.random.default_rng(seed)
    groups, c = [], 0
    for k in cards:
        groups.append(cg.ColGroupDDC(list(range(c, c + width)), rng.standard_normal((k, width)),
                                     MapToFactory.create_from(rng.integers(0, k, nRows), k)))
        c += width
    if const:
        groups.append(cg.ColGroupConst([c], [[0.75]]))
        c += 1
    return CompressedMatrixBlock(nRows, c, groups)


def _check(cmb, ks=(1,), qs=(1,), chain=True, seed=0):
    X = dense_of(cmb)
    aX = np.abs(X)
    n, m = X.shape
    rng = np.random.default_rng(seed)
    for k in ks:
        V = rng.standard_normal((m, k))
        got = CLALibRightMultBy.rightMultByMatrix(cmb, V)
        assert rel_err(got, X @ V, aX @ np.abs(V) + 1e-300) < TOL, ("rmm", k)
        assert got.nnz == np.count_nonzero(got)
    for q in qs:
        Y = rng.standard_normal((q, n))
        got = CLALibLeftMultBy.leftMultByMatrix(cmb, Y)
        assert rel_err(got, Y @ X, np.abs(Y) @ aX + 1e-300) < TOL, ("lmm", q)
        assert got.nnz == np.count_nonzero(got)
    if chain:
        v, w = rng.standard_normal(m), rng.standard_normal(n)
        s = aX.T @ (np.abs(w) * (aX @ np.abs(v))) + 1e-300
        assert rel_err(CLALibMMChain.mmChain(cmb, v, w, CHAIN_XtwXv).ravel(), X.T @ (w * (X @ v)), s) < 10 * TOL
        s = aX.T @ (aX @ np.abs(v)) + 1e-300
        assert rel_err(CLALibMMChain.mmChain(cmb, v).ravel(), X.T @ (X @ v), s) < 10 * TOL


@pytest.mark.parametrize("nRows", [1, 31, 33, 1025, 4095, 4096])
def test_short_blocks_every_group_type(nRows):
    """The one-kernel products on blocks below 4096 rows, and the first row count above them."""
    kinds = datagen.KINDS + ("ddcfor", "ddc2", "ole", "rle", "sdc")
    cmb = datagen.random_cmb(31 * nRows + 7, nRows, kinds).to_device()
    _check(cmb, ks=(1, 3, 5, 8, 9), qs=(1, 2, 4, 5))
    cmb.free()


@pytest.mark.parametrize("nCols", [450, 900])
def test_short_blocks_wide_right_operand(nCols):
    """V beyond what travels with the launch (448 values) and beyond what fits shared memory (6144)."""
    cmb = _ddc(77, [5] * nCols, nCols, const=True).to_device()
    _check(cmb, ks=(1, 8), chain=False)
    cmb.free()


@pytest.mark.parametrize("nRows,nCols", [(4097, 16), (4127, 17), (5000, 112), (5000, 113), (9000, 240), (300007, 20)])
@pytest.mark.parametrize("card", [2, 7, 16, 256])
def test_byte_map_units(nRows, nCols, card):
    """Column-per-lane kernels: last unit partly filled, one unit more than the fused chain takes, several chunks, joint
    slots (tall blocks of small dictionaries), bit maps; a constant column."""
    cmb = _ddc(nRows, [card] * nCols, nRows + nCols + card, const=nCols % 2 == 1).to_device()
    _check(cmb, qs=(1, 2, 5, 8, 9))
    cmb.free()


def test_joint_slots_of_uneven_dictionaries():
    """Mixed-radix joint ids: one to eight groups per slot, single tuples, co-coded columns."""
    cards = [1, 1, 2, 2, 2, 3, 3, 5, 7, 11, 13, 16, 17, 40, 128, 255, 256] + [2] * 20 + [3] * 15
    for width in (1, 2):
        cmb = _ddc(300001, cards, 5 + width, width=width).to_device()
        _check(cmb)
        cmb.free()


@pytest.mark.parametrize("cards", [[16] * 33, [16] * 40, [16] * 42, [6] * 51, [2] * 144, [16] * 195, [200] * 20 + [16] * 40, [2, 128] * 20])
def test_joint_slots_behind_the_last_unit(cards):
    """Joint slots by rows: one, four and none behind the last whole unit; parts of one and of several groups; several chunks;
    slots of one group. Inf and NaN entries stay in their rows, also those of the slots that go by rows."""
    cmb = _ddc(300001, cards, len(cards)).to_device()
    _check(cmb, chain=False)
    cmb.free()
    rng = np.random.default_rng(3)
    groups = []
    for c, k in enumerate(cards):
        d = rng.standard_normal((k, 1))
        ids = rng.integers(0, k - 1, 300001)
        if c % 16 in (0, 7):
            d[k - 1] = np.inf if c % 2 else np.nan
            ids[rng.integers(0, 300001, 20)] = k - 1
        groups.append(cg.ColGroupDDC([c], d, MapToFactory.create_from(ids, k)))
    cmb = CompressedMatrixBlock(300001, len(cards), groups).to_device()
    X = dense_of(cmb)
    v = rng.standard_normal(len(cards))
    got = np.asarray(CLALibRightMultBy.rightMultByMatrix(cmb, v)).ravel()
    fine = np.isfinite(X).all(axis=1)
    assert 0 < fine.sum() < 300001
    assert np.array_equal(np.isfinite(got), fine)
    assert rel_err(got[fine], X[fine] @ v, np.abs(X[fine]) @ np.abs(v)) < TOL
    cmb.free()


@pytest.mark.parametrize("nRows", [5000, 300007])
def test_non_finite_values_stay_in_their_rows(nRows):
    """Inf and NaN dictionary entries reach the rows that hold them and no other (the row sums of neighbouring rows are
    formed by one matrix product)."""
    rng = np.random.default_rng(1)
    groups = []
    for c in range(40):
        d = rng.standard_normal((100, 1))
        if c % 13 == 0:
            d[5], d[6] = np.inf, np.nan
        ids = rng.integers(7, 100, nRows)
        hit = rng.random(nRows) < 0.01
        ids[hit] = rng.integers(5, 7, int(hit.sum()))
        groups.append(cg.ColGroupDDC([c], d, MapToFactory.create_from(ids, 100)))
    cmb = CompressedMatrixBlock(nRows, 40, groups).to_device()
    X = dense_of(cmb)
    v = rng.standard_normal(40)
    with np.errstate(invalid="ignore"):
        want = X @ v
    got = np.asarray(CLALibRightMultBy.rightMultByMatrix(cmb, v)).ravel()
    fine = np.isfinite(X).all(axis=1)
    assert 0 < fine.sum() < nRows
    assert np.array_equal(np.isfinite(got), fine)
    assert rel_err(got[fine], want[fine], np.abs(X[fine]) @ np.abs(v)) < TOL
    cmb.free()


@pytest.mark.parametrize("nRows", [4127, 40001])
def test_left_product_of_non_finite_values(nRows):
    """Inf in the left vector makes Inf, not NaN, of columns of one sign, whichever rows share its products with zeros; NaN
    and the ragged last rows likewise."""
    rng = np.random.default_rng(nRows)
    groups = [cg.ColGroupDDC([c], rng.uniform(0.5, 1.0, (9, 1)), MapToFactory.create_from(rng.integers(0, 9, nRows), 9)) for c in range(40)]
    cmb = CompressedMatrixBlock(nRows, 40, groups).to_device()
    for row in (0, 3, 18, nRows - 1, nRows - 40):
        for value in (np.inf, -np.inf, np.nan):
            y = rng.standard_normal((1, nRows))
            y[0, row] = value
            got = np.asarray(CLALibLeftMultBy.leftMultByMatrix(cmb, y)).ravel()
            assert np.isnan(got).all() if np.isnan(value) else (got == value).all()
    cmb.free()


@pytest.mark.parametrize("nRows", [33, 5000])
@pytest.mark.parametrize("nCols", [127, 129, 160, 257])
def test_self_product_blocks(oracle, nRows, nCols):
    """t(X) X with and without SDC / RLE columns around the edges of the 128 x 128 blocks and their 32 x 32 tiles."""
    for kinds in (("ddc",) * nCols, ("ddc", "sdc", "rle") * (nCols // 3) + ("ddc",) * (nCols % 3)):
        cmb = datagen.random_cmb(nCols + nRows, nRows, kinds).to_device()
        X = dense_of(cmb)
        got = CLALibTSMM.leftMultByTransposeSelf(cmb)
        assert rel_err(got, oracle.dense_tsmm_ld(X), np.abs(X).T @ np.abs(X) + 1e-300) < TOL
        assert np.array_equal(got, got.T)
        cmb.free()


def _six_kinds(nRows, nCols, by_kind):
    """Byte and wide maps, listed rows without and with a default tuple, runs, dense columns; all of them of modest spread."""
    rng = np.random.default_rng(nCols)
    kinds = ["ddc", "sdc", "default", "rle", "unc", "wide"]
    groups = []
    for c in range(nCols):
        k = kinds[c * 6 // nCols if by_kind else c % 6]
        if k == "ddc":
            n = int(rng.integers(2, 40))
            groups.append(cg.ColGroupDDC([c], rng.standard_normal((n, 1)), MapToFactory.create_from(rng.integers(0, n, nRows), n)))
        elif k == "wide":
            groups.append(cg.ColGroupDDC([c], rng.uniform(-1, 1, (400, 1)), MapToFactory.create_from(rng.integers(0, 400, nRows), 400)))
        elif k in ("sdc", "default"):
            rows = np.flatnonzero(rng.random(nRows) < 0.1)
            ids = MapToFactory.create_from(rng.integers(0, 5, rows.size), 5)
            d, off = rng.standard_normal((5, 1)), OffsetFactory.createOffset(rows)
            groups.append(cg.ColGroupSDCZeros([c], nRows, d, off, ids) if k == "sdc" else
                          cg.ColGroupSDC([c], nRows, d, np.array([0.3]), off, ids))
        elif k == "rle":
            ends = np.minimum(np.cumsum(rng.geometric(0.01, size=nRows // 30)), nRows)
            starts = np.concatenate([[0], ends[:-1]])
            keep = ends > starts
            starts, ends = starts[keep], ends[keep]
            ends[-1] = nRows
            groups.append(cg.ColGroupRLE.from_runs([c], rng.standard_normal((9, 1)), starts, ends - starts, rng.integers(0, 9, starts.size), nRows))
        else:
            groups.append(cg.ColGroupUncompressed([c], rng.standard_normal((nRows, 1))))
    return CompressedMatrixBlock(nRows, nCols, groups)


def _entries_in_digits(got, want, X, oracles):
    """Every entry for itself: 2^-50 of the sum of its terms' magnitudes is what a block may lose that is taken in digits."""
    assert (np.abs(got - want) <= 2.0**-50 * (np.abs(X).T @ np.abs(X)) + oracles + 2.0**-52 * np.abs(want)).all()


@pytest.mark.parametrize("nRows,nCols", [(11364, 176), (8193, 255), (20011, 257), (40001, 384), (4096, 500)])
@pytest.mark.parametrize("by_kind", [True, False])
def test_self_product_in_digits(oracle, nRows, nCols, by_kind):
    """t(X) X by 8-bit digits, straight from the columns and from decompressed rows: smallest sizes, blocks of 128 columns with
    few and many left over, row remainders. What is lost lies 55 bits behind a column's power of two 2^e (2^-56 of it
    per cell at most) and behind weight 7 (five products of digits below 2^14 in units of 2^-78, and what follows); then the
    result is rounded. Integers: the same bits from every call."""
    cmb = _six_kinds(nRows, nCols, by_kind).to_device()
    X = dense_of(cmb)
    got = np.array(CLALibTSMM.leftMultByTransposeSelf(cmb))
    want = oracle.dense_tsmm_ld(X)
    e = np.exp2(np.ceil(np.log2(np.abs(X).max(axis=0) / 0.99)))
    a = np.abs(X).sum(axis=0)
    lost = 2.0**-56 * (np.outer(e, a) + np.outer(a, e)) + nRows * 2.0**-60 * np.outer(e, e)
    oracles = nRows * 2.0**-64 * (np.abs(X).T @ np.abs(X))  # long double, one sum after the other
    assert (np.abs(got - want) <= lost + oracles + 2.0**-52 * np.abs(want)).all()
    norms = np.sqrt(np.outer(np.diag(want), np.diag(want)))
    assert (np.abs(got - want) / norms).max() < 1e-15  # (the FP64 products: 4e-15 to 2e-14)
    _entries_in_digits(got, want, X, oracles)
    assert np.array_equal(got, got.T)
    assert np.array_equal(got, np.array(CLALibTSMM.leftMultByTransposeSelf(cmb)))
    cmb.free()


def _self_product_in_digits(oracle, cmb):
    X = dense_of(cmb)
    got = np.array(CLALibTSMM.leftMultByTransposeSelf(cmb))
    want = oracle.dense_tsmm_ld(X)
    norms = np.sqrt(np.outer(np.diag(want), np.diag(want)))
    assert (np.abs(got - want) / norms).max() < 1e-15
    _entries_in_digits(got, want, X, X.shape[0] * 2.0**-64 * (np.abs(X).T @ np.abs(X)))
    assert np.array_equal(got, got.T)
    assert np.array_equal(got, np.array(CLALibTSMM.leftMultByTransposeSelf(cmb)))


@pytest.mark.parametrize("nRows", [16384, 16399, 20001])
@pytest.mark.parametrize("cards,width", [([7] * 129, 1), ([2, 256, 100] * 50, 1), ([400, 1600, 3] * 48, 1), ([9, 300] * 40, 2)])
def test_self_product_of_dense_maps_in_digits(oracle, nRows, cards, width):
    """Bit, byte and 16-bit maps, the longest tables, co-coded columns, a lane's last rows, part units of 16 columns."""
    cmb = _ddc(nRows, cards, nRows + len(cards), width=width).to_device()
    _self_product_in_digits(oracle, cmb)
    cmb.free()


def test_self_product_in_digits_of_many_rows():
    """More rows than one round of 64-bit sums takes: 1' (X'X) 1 = |X 1|^2, and the square sums of single columns."""
    torch = pytest.importorskip("torch")
    from systemds_b200.mapping import MAP_BYTE, DeviceMap
    n, cols = 5_000_017, 130
    gen = torch.Generator(device="cuda")
    gen.manual_seed(4)
    rng = np.random.default_rng(4)
    groups, ones, squares = [], torch.zeros(n, dtype=torch.float64, device="cuda"), []
    for c in range(cols):
        ids = torch.randint(0, 50, (n,), dtype=torch.uint8, device="cuda", generator=gen)
        d = rng.standard_normal((50, 1))
        x = torch.from_numpy(d.ravel()).cuda()[ids.long()]
        ones += x
        squares.append(float((x * x).sum()))
        groups.append(cg.ColGroupDDC([c], d, DeviceMap(MAP_BYTE, n, 50, ids.data_ptr(), n, owner=ids)))
    torch.cuda.synchronize()
    cmb = CompressedMatrixBlock(n, cols, groups).to_device()
    got = np.array(CLALibTSMM.leftMultByTransposeSelf(cmb))
    assert np.allclose(np.diag(got), squares, rtol=1e-12, atol=0)
    assert abs(got.sum() - float((ones * ones).sum())) <= 1e-12 * np.abs(got).sum()
    assert np.array_equal(got, got.T)
    cmb.free()


def test_self_product_of_integers_in_digits():
    """Integers of up to 24 bits: nothing is lost, to the last bit of sums below 2^53."""
    rng = np.random.default_rng(2)
    groups = [cg.ColGroupDDC([c], rng.integers(-2**16, 2**16, (9, 1)).astype(float) * (2.0**8 if c % 3 else 2.0**-20),
                             MapToFactory.create_from(rng.integers(0, 9, 12000), 9)) for c in range(200)]
    cmb = CompressedMatrixBlock(12000, 200, groups).to_device()
    X = dense_of(cmb)
    s = np.where(np.arange(200) % 3, 2.0**-8, 2.0**20)
    Z = (X * s).astype(np.int64)
    assert np.array_equal(np.array(CLALibTSMM.leftMultByTransposeSelf(cmb)), (Z.T @ Z).astype(float) / np.outer(s, s))
    cmb.free()


@pytest.mark.parametrize("values", [[1e6] + [1.0] * 8, [np.inf] + [1.0] * 8, [np.nan] + [1.0] * 8, [1e-200, 2e-200] + [1e-200] * 7, [0.0] * 9])
def test_self_product_without_digits(values):
    """One column whose values stand out too far, are not finite or too small, or all zero: the products in double precision, or
    digits that are all zero."""
    rng = np.random.default_rng(1)
    groups = [cg.ColGroupDDC([c], rng.standard_normal((9, 1)), MapToFactory.create_from(rng.integers(0, 9, 12000), 9)) for c in range(199)]
    ids = rng.integers(1, 9, 12000)
    ids[17] = 0
    groups.append(cg.ColGroupDDC([199], np.array(values).reshape(-1, 1), MapToFactory.create_from(ids, 9)))
    cmb = CompressedMatrixBlock(12000, 200, groups).to_device()
    X = dense_of(cmb)
    got = np.array(CLALibTSMM.leftMultByTransposeSelf(cmb))
    with np.errstate(invalid="ignore"):
        want, s = X.T @ X, np.abs(X).T @ np.abs(X)
    fine = np.isfinite(want)
    assert np.array_equal(np.isfinite(got), fine)
    assert (np.abs(got[fine] - want[fine]) <= TOL * s[fine] + 1e-320).all()
    cmb.free()


def _two_scales(nRows, small, kinds, by_kind):
    """200 columns, of every kind some a that are about 1 in the first half of the rows and about `small` in the others, and some b
    that are about 1 in the others alone; small = 0: a is 1 in one row and 1e-18 in the others, b not zero in the others."""
    rng = np.random.default_rng(nRows)
    first = np.arange(nRows) < (nRows // 2 if small else 1)
    groups = []
    for c in range(200):
        k = kinds[c * len(kinds) // 200 if by_kind else c % len(kinds)]
        d = np.concatenate([rng.uniform(0.9, 1.1, 3), rng.uniform(0.9, 1.1, 3) * (small or 1e-18)] if c % 20 < 10 else [[0.0], rng.uniform(0.9, 1.1, 5)])
        if c % 20 >= 10:
            ids = np.where(first, 0, rng.integers(1, 6, nRows))
        elif small:
            ids = np.where(first, rng.integers(0, 3, nRows), rng.integers(3, 6, nRows))
        else:
            d[:3] = 1.0
            ids = np.where(first, 0, rng.integers(3, 6, nRows))
        d = d.reshape(-1, 1)
        if k == "ddc":
            groups.append(cg.ColGroupDDC([c], d, MapToFactory.create_from(ids, 6)))
        elif k == "unc":
            groups.append(cg.ColGroupUncompressed([c], d[ids]))
        elif k == "sdc":  # the value of the first rows is the default
            rows = np.flatnonzero(~first)
            off, m = OffsetFactory.createOffset(rows), MapToFactory.create_from(ids[rows], 6)
            groups.append(cg.ColGroupSDCZeros([c], nRows, d, off, m) if d[0, 0] == 0.0 else
                          cg.ColGroupSDC([c], nRows, d, d[0].copy(), off, m))
        else:
            ids = np.where(first, ids[0], np.repeat(ids[::-1][:nRows // 50 + 1], 50)[:nRows][::-1])
            starts = np.flatnonzero(np.diff(ids, prepend=-1))
            groups.append(cg.ColGroupRLE.from_runs([c], d, starts, np.diff(starts, append=nRows), ids[starts], nRows))
    return CompressedMatrixBlock(nRows, 200, groups)


@pytest.mark.parametrize("small", [1e-6, 1e-9, 1e-12, 1e-18, 0])
@pytest.mark.parametrize("kinds,by_kind", [(["ddc"], True), (["ddc", "sdc", "rle", "unc"], True), (["ddc", "sdc", "rle", "unc"], False)])
def test_self_product_of_columns_of_two_scales(oracle, small, kinds, by_kind):
    """Entries whose terms are far below their columns' largest magnitudes, as precise as the others: dense maps, columns by kind,
    decompressed rows. The bound is the sum's, a rounding of 2^-53 per four rows, and the oracle's."""
    nRows = 20011
    cmb = _two_scales(nRows, small, kinds, by_kind)
    X = dense_of(cmb)
    cmb.to_device()
    want, s = oracle.dense_tsmm_ld(X), np.abs(X).T @ np.abs(X)
    for _ in range(2):
        got = np.array(CLALibTSMM.leftMultByTransposeSelf(cmb))
        assert (np.abs(got - want) <= nRows * 2.0**-55 * s).all(), (np.abs(got - want) / (s + 1e-300)).max()
    cmb.free()


@pytest.mark.parametrize("unused", [1e7, 1e18, 1e100])
@pytest.mark.parametrize("kind", ["ddc", "sdc", "default", "rle"])
def test_self_product_with_unused_tuples(oracle, kind, unused):
    """A tuple that no row has lies far above the cells (bounds of the columns come from the dictionaries): a dense map and a column
    of `kind` have one, in a block of dense maps for `ddc`."""
    rng = np.random.default_rng(12)
    n, groups = 12003, []
    for c in range(200):
        d = rng.uniform(0.5, 1.0, (6, 1)) * (1.0 if c % 2 else -1.0)
        if c in (3, 140):
            d[5] = unused
        ids = rng.integers(0, 5, n)
        rows = np.flatnonzero(rng.random(n) < 0.4)
        if kind == "ddc" or c < 100:
            groups.append(cg.ColGroupDDC([c], d, MapToFactory.create_from(ids, 6)))
        elif kind == "rle":
            starts = np.flatnonzero(np.diff(ids, prepend=-1))
            groups.append(cg.ColGroupRLE.from_runs([c], d, starts, np.diff(starts, append=n), ids[starts], n))
        elif kind == "sdc":
            groups.append(cg.ColGroupSDCZeros([c], n, d, OffsetFactory.createOffset(rows), MapToFactory.create_from(ids[rows], 6)))
        else:  # where every row is listed, the default tuple is the unused one
            every = np.arange(n) if c == 140 else rows
            groups.append(cg.ColGroupSDC([c], n, d[:5], d[5].copy(), OffsetFactory.createOffset(every), MapToFactory.create_from(ids[every], 5)))
    cmb = CompressedMatrixBlock(n, 200, groups)
    X = dense_of(cmb)
    assert np.abs(X).max() <= 1.0
    cmb.to_device()
    want, s = oracle.dense_tsmm_ld(X), np.abs(X).T @ np.abs(X)
    for _ in range(2):
        got = np.array(CLALibTSMM.leftMultByTransposeSelf(cmb))
        assert (np.abs(got - want) <= n * 2.0**-55 * s).all(), (np.abs(got - want) / (s + 1e-300)).max()
    cmb.free()


@pytest.mark.parametrize("i,j", [(0, 1), (7, 131), (127, 128), (130, 259), (258, 259)])
@pytest.mark.parametrize("row", [0, 16383, 50002])
def test_self_product_with_one_small_term(i, j, row):
    """One entry of the result has a single term, far below what its columns hold elsewhere: the product itself, wherever the
    pair of columns and the row lie."""
    rng = np.random.default_rng(i + j)
    n, groups = 50003, []
    for c in range(260):
        ids, d = rng.integers(1, 9, n), rng.uniform(0.5, 1.0, 9)
        ids[row], d[0] = 0, 0.7
        if c == i:
            d[0] = 3.3e-17
        elif c == j:
            d[1:] = 0.0
        groups.append(cg.ColGroupDDC([c], d.reshape(-1, 1), MapToFactory.create_from(ids, 9)))
    cmb = CompressedMatrixBlock(n, 260, groups).to_device()
    for _ in range(2):
        got = np.array(CLALibTSMM.leftMultByTransposeSelf(cmb))
        assert got[i, j] == got[j, i] == 3.3e-17 * 0.7
    cmb.free()


@pytest.mark.parametrize("nRows", [1, 255, 257, 1040, 5001])
@pytest.mark.parametrize("nCols", [31, 33, 530])
def test_decompress_columns(nRows, nCols):
    """Decompress with the columns of a CTA of every kind, row remainders and part blocks: the cells are the registered
    values."""
    kinds = ("ddc", "sdcz", "rle", "unc", "ddc_bit", "sdc", "const", "empty", "ole", "sdcs")
    kinds = kinds * (nCols // 11) + ("ddc",) * (nCols % 11)
    cmb = datagen.random_cmb(nRows + nCols, nRows, kinds).to_device()
    assert np.array_equal(np.array(CLALibDecompress.decompress(cmb)), dense_of(cmb))
    cmb.free()


@pytest.mark.parametrize("stretches", [5, 8, 9, 11, 13, 17])
def test_decompress_columns_in_rows_of_ctas(stretches):
    """A kind per 32 columns, the last 32 cut short: one CTA along a row, several that come out even, and with warps left over."""
    nRows, nCols = (4 << 20) // (stretches * 32 - 5) + 16, stretches * 32 - 5
    cmb = datagen.random_cmb(stretches, nRows, [("ddc", "sdcz", "rle", "unc")[c // 32 % 4] for c in range(nCols)])
    X = dense_of(cmb)
    cmb.to_device()
    for _ in range(3):  # by columns from the second call on
        assert np.array_equal(np.array(CLALibDecompress.decompress(cmb)), X)
    cmb.free()


@pytest.mark.parametrize("nRows", [4096, 4127, 4161])
@pytest.mark.parametrize("kinds", ["bytes", "chars", "mixed", "sparse", "cocoded"])
def test_wide_right_operand(nRows, kinds):
    """X %*% V around the tile widths (8, 16, 24, 32 columns, two slices) and row remainders: several chunks of columns,
    padding columns of every kind, dictionaries too large to stay resident, odd column counts, no dense column at all,
    SDC and RLE groups of two columns (tables instead of rows of V)."""
    if kinds == "bytes":
        cmb = _ddc(nRows, [256] * 130 + [2, 2, 3], 3, const=True)
    elif kinds == "chars":
        cmb = _ddc(nRows, [300, 1000, 4096, 5000] * 3 + [9], 4)
    elif kinds == "mixed":
        cmb = datagen.random_cmb(nRows, nRows, datagen.KINDS + ("unc", "ddc2", "ddc_char", "rle", "sdcz"))
    elif kinds == "cocoded":
        rng = np.random.default_rng(nRows)
        cmb = CompressedMatrixBlock(nRows, 9, [datagen.random_group(k, c, nRows, rng) for k, c in (
            ("sdc", [0, 1]), ("rle", [2, 3]), ("sdcz", [4]), ("ddc", [5]), ("rle", [6]), ("sdcs", [7, 8]))])
    else:
        cmb = datagen.random_cmb(nRows, nRows, ("sdc", "sdcz", "rle", "sdcs", "const", "rle"))
    cmb.to_device()
    _check(cmb, ks=(2, 3, 7, 8, 9, 16, 17, 24, 25, 32, 33, 64, 65), qs=(2, 3, 8, 9), chain=False)
    cmb.free()


@pytest.mark.parametrize("nRows", [16384, 17001, 74003, 120001])
@pytest.mark.parametrize("longest", [257, 1601, 6400, 6401])
def test_products_with_tables_of_16_bit_maps(nRows, longest):
    """Sixteen, eight and four columns per CTA, a table that stays in global memory, co-coded and constant columns."""
    cmb = _ddc(nRows, [300, 1000, 257] * 6 + [longest, 9], longest, const=True, width=2 if longest == 1601 else 1).to_device()
    _check(cmb, ks=(1,), qs=(1, 2, 5, 9))
    cmb.free()


def _sdc(nRows, dens, card, default, seed, rows=None):
    """An SDC column with listed rows of the given density (or exactly `rows`)."""
    rng = np.random.default_rng(seed)
    ids = np.full(nRows, -1, np.int32)
    mask = rng.random(nRows) < dens if rows is None else np.isin(np.arange(nRows), rows)
    ids[mask] = rng.integers(0, card, int(mask.sum()))
    return lambda c: cg.sdc_from_row_ids([c], rng.standard_normal((card, 1)), ids, rng.standard_normal(1) if default else None)


def _by_kind(nRows):
    """A kind per 32 columns, as the decompress by columns wants them: offset streams with 8- and 16-bit deltas, gaps beyond
    their range, dense lists, none, one or two listed rows (also at the edges of 64-row pieces), one tuple only; short and
    long runs, rows without a run; byte and bit maps; dense columns; a few long tables and two-column groups."""
    rng = np.random.default_rng(nRows)
    groups, c = [], 0

    def add(make, width=1):
        nonlocal c
        groups.append(make(c) if width == 1 else make(list(range(c, c + width))))
        c += width

    last = nRows - 1
    for i, (dens, card) in enumerate([(0.05, 8), (0.0004, 8), (0.5, 3), (0.3, 300), (0.02, 1), (0.999, 2)] * 5):
        add(_sdc(nRows, dens, card, i % 2, i))
    add(_sdc(nRows, 0, 3, False, 1, rows=[63, 64, 1023, 1024, last]))
    add(_sdc(nRows, 0, 3, True, 2, rows=[last - 1]))
    for rows in ([0], [last], [0, last], [63, 64], [64], [1023, 1024], [5000, last], [2]):
        add(_sdc(nRows, 0, 2, len(rows) == 1, 3, rows=rows))
    for i in range(24):
        add(_sdc(nRows, 0.05, 5, i % 2, 100 + i))
    for i in range(32):
        add(lambda c: datagen.random_group("rle", [c], nRows, rng))
    for i in range(32):
        add(lambda c: datagen.random_group("ddc_bit" if i % 3 else "ddc", [c], nRows, rng))
    for i in range(16):
        add(lambda cs: datagen.random_group("ddc2", cs, nRows, rng), 2)
    for i in range(4):
        add(lambda cs: datagen.random_group("unc", cs, nRows, rng), 8)
    for i in range(31):
        add(lambda c: datagen.random_group("const" if i % 2 else "empty", [c], nRows, rng))
    for i in range(2):
        add(lambda c: datagen.random_group("ddc_char", [c], nRows, rng))
    return CompressedMatrixBlock(nRows, c, groups)


@pytest.mark.parametrize("nRows", [18817, 19455, 70001, 93313])
def test_decompress_by_columns(nRows):
    """From four million cells on, columns sorted by kind; the first call on a block (by columns from 20 million cells on) and
    a repeated one: the cells are the registered values, also in the row chunks of a self product, and the handle takes no
    more memory than one word per listed row and a record per column."""
    cmb = _by_kind(nRows)
    assert nRows * cmb.clen >= 4 << 20
    X = dense_of(cmb)
    cmb.to_device()
    held = cmb.stats()["device_bytes"]
    for _ in range(2):
        assert np.array_equal(np.array(CLALibDecompress.decompress(cmb)), X)
    listed = sum(g._indexes.getSize() for g in cmb.getColGroups() if hasattr(g, "_indexes"))
    assert cmb.stats()["device_bytes"] - held <= 4 * listed + 64 * cmb.clen + 256
    got = CLALibTSMM.leftMultByTransposeSelf(cmb)
    assert rel_err(got, X.T @ X, np.abs(X).T @ np.abs(X) + 1e-300) < TOL
    _check(cmb, ks=(1, 3), chain=False)
    assert np.array_equal(np.array(CLALibDecompress.decompress(cmb)), X)
    cmb.free()


def test_decompress_by_columns_with_references():
    """Columns held by a group and by the constant group of its reference tuple: a cell is the sum of both. Such a block adds
    the folded constants in every column: c + (d - c) for an SDC column with default c. The difference and the sum round
    once each, so a cell is off by at most eps / 2 times |d - c| + |d| <= eps (|d| + |c|)."""
    nRows, rng = 18817, np.random.default_rng(3)
    cmb = _by_kind(nRows)
    groups, c = list(cmb.getColGroups()), cmb.clen
    for i in range(63):
        groups.append(datagen.random_group("sdcfor" if i < 32 else "ddcfor", [c], nRows, rng))
        c += 1
    cmb = CompressedMatrixBlock(nRows, c, groups)
    X, scale = dense_of(cmb), abs_dense_of(cmb) + 1e-300
    for g in groups:
        if getattr(g, "_defaultTuple", None) is not None:
            scale[:, g.getColIndices()] += np.abs(g._defaultTuple)
    cmb.to_device()
    for _ in range(2):
        assert rel_err(np.array(CLALibDecompress.decompress(cmb)), X, scale) <= 1.01 * np.finfo(float).eps
    cmb.free()

def _runs_and_lists(nRows, nCols):
    """Runs and lists whose entries lie at the edges of sixteen rows: single rows, neighbouring runs, runs over many groups of
    sixteen, full and empty groups, entries in the last row."""
    rng = np.random.default_rng(nRows)
    groups = []
    for c in range(nCols):
        if c < nCols // 2:
            cuts = np.unique(np.concatenate([np.arange(16, nRows, 16) + rng.integers(-1, 2, (nRows - 1) // 16), np.arange(64 * (c % 5), 64 * (c % 5) + 40),
                                             [0, nRows - 1, nRows]]))
            cuts = cuts[(cuts == 0) | (cuts >= nRows - 1) | (rng.random(cuts.size) < [1.0, 0.5, 0.05][c % 3])]
            starts, ends = cuts[:-1], cuts[1:]
            keep = rng.random(starts.size) < [1.0, 0.7][c % 2]
            keep[-1] = True
            starts, lens = starts[keep], (ends - starts)[keep]
            groups.append(cg.ColGroupRLE.from_runs([c], rng.standard_normal((9, 1)), starts, lens, rng.integers(0, 9, starts.size), nRows))
        else:
            p = np.repeat(rng.choice([0.0, 0.06, 0.5, 1.0], nRows // 16 + 1), 16)[:nRows]
            rows = np.flatnonzero((rng.random(nRows) < p) | np.isin(np.arange(nRows), [0, 15, 16, nRows - 1]))
            ids, d = MapToFactory.create_from(rng.integers(0, 5, rows.size), 5), rng.standard_normal((5, 1))
            off = OffsetFactory.createOffset(rows)
            groups.append(cg.ColGroupSDCZeros([c], nRows, d, off, ids) if c % 2 else cg.ColGroupSDC([c], nRows, d, np.array([0.3]), off, ids))
    return CompressedMatrixBlock(nRows, nCols, groups)


@pytest.mark.parametrize("nRows,nCols", [(33001, 192), (16384, 289), (14001, 350), (9999, 576)])
def test_runs_and_lists_by_sixteen_rows(oracle, nRows, nCols):
    """Decompress copies values, so it is exact; t(X) X then reads the same walks as digits. CTAs of 6, 5, 11 and 6 warps."""
    cmb = _runs_and_lists(nRows, nCols)
    X = dense_of(cmb)
    cmb.to_device()
    for _ in range(2):
        assert np.array_equal(np.array(CLALibDecompress.decompress(cmb)), X)
    _self_product_in_digits(oracle, cmb)
    cmb.free()


def test_decompress_first_called_in_a_capture():
    """A captured call leaves no plan that only its replay would fill: direct calls and replays after it are right."""
    import torch
    from systemds_b200 import native
    cmb = _by_kind(93313)
    X = torch.from_numpy(dense_of(cmb)).cuda()
    cmb.to_device()
    lib, h = native.lib(), cmb.handle()
    out, stream, graph = torch.empty_like(X), torch.cuda.Stream(), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream):
        native.check(lib.cla_decompress_dev(h, out.data_ptr(), stream.cuda_stream))
    with torch.cuda.stream(stream):
        for call in (lambda: native.check(lib.cla_decompress_dev(h, out.data_ptr(), stream.cuda_stream)), graph.replay) * 2:
            out.zero_()
            call()
            stream.synchronize()
            assert torch.equal(out, X)
    del graph
    cmb.free()


@pytest.mark.parametrize("by_kind", [True, False])
def test_self_product_first_called_in_a_capture(by_kind):
    """A captured first call cannot look at the block: its replay does the sums in double precision, direct calls before and
    after a replay in digits where the block suits them. A call captured later replays what direct calls give."""
    import torch
    from systemds_b200 import native
    cmb = _six_kinds(20011, 257, by_kind)
    X = torch.from_numpy(dense_of(cmb)).cuda()
    want, bound = X.T @ X, 2 * 20011 * 2.0**-55 * (X.abs().T @ X.abs())
    cmb.to_device()
    lib, h = native.lib(), cmb.handle()
    out, stream = torch.empty_like(want), torch.cuda.Stream()
    first, later = torch.cuda.CUDAGraph(), torch.cuda.CUDAGraph()

    def call():
        native.check(lib.cla_tsmm_dev(h, out.data_ptr(), stream.cuda_stream))

    def result(f):
        with torch.cuda.stream(stream):
            out.zero_()
            f()
            stream.synchronize()
            assert ((out - want).abs() <= bound).all()
            return out.clone()

    torch.cuda.synchronize()
    with torch.cuda.graph(first, stream=stream, capture_error_mode="relaxed"):  # (the call grows its scratch)
        call()
    result(first.replay)
    direct = result(call)
    result(first.replay)
    with torch.cuda.graph(later, stream=stream):
        call()
    assert torch.equal(result(later.replay), direct) and torch.equal(result(call), direct)
    del first, later
    cmb.free()


@pytest.mark.parametrize("nCols", [128, 129, 300, 448, 449])
@pytest.mark.parametrize("nRows", [77, 1000])
def test_short_blocks_with_v_in_the_launch(nRows, nCols):
    """A host-buffer product whose V travels with the launch: the last count of the small argument, the first and last of
    the large one, and the first that is read from the mailbox instead."""
    cmb = _ddc(nRows, [5] * (nCols - 1), nCols, const=True).to_device()
    assert cmb.clen == nCols
    _check(cmb, qs=(1,))
    cmb.free()


@pytest.mark.parametrize("longest", [6400, 6401])
@pytest.mark.parametrize("extra", [-1, 0, 33])
def test_right_product_with_the_longest_tables(longest, extra):
    """X %*% v with tables of four columns per CTA: taken from half a table's rows per SM on, which the longest table that
    fits needs most rows for; one tuple more, and the column stays with the other kernel."""
    import torch
    nRows = torch.cuda.get_device_properties(0).multi_processor_count * 3200 + extra
    cmb = _ddc(nRows, [longest, 300, 257, longest, 1000, 512], longest + extra, const=True).to_device()
    _check(cmb, ks=(1,), qs=(1, 2))
    cmb.free()
