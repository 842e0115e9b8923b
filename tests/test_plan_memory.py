"""Products of handles whose plans find no memory: every call takes the kernels that work on the registered arrays and
gives the same products, the first time and when repeated."""
import numpy as np
import pytest

from systemds_b200 import CompressedMatrixBlock, datagen, native
from systemds_b200.cmb import CLALibDecompress, CLALibTSMM
from systemds_b200 import colgroup as cg
from systemds_b200.mapping import MapToFactory
from systemds_b200.native import check
from tests.test_kernel_edges import _by_kind, _check, _ddc
from tests.util import TOL, dense_of, rel_err


def _cocoded(nRows):
    rng = np.random.default_rng(nRows)
    return CompressedMatrixBlock(nRows, 13, [datagen.random_group(k, c, nRows, rng) for k, c in (
        ("sdc", [0, 1]), ("rle", [2, 3]), ("sdcz", [4]), ("ddc", [5]), ("rle", [6]), ("sdcs", [7, 8]), ("unc", [9, 10, 11]),
        ("ddc_char", [12]))])


def _wide_dense(nRows):  # more uncompressed columns than a block has threads
    rng = np.random.default_rng(nRows)
    return CompressedMatrixBlock(nRows, 523, [datagen.random_group(k, c, nRows, rng) for k, c in (
        ("sdcz", [0]), ("unc", list(range(1, 521))), ("rle", [521, 522]))])


BLOCKS = {
    "short": lambda: datagen.random_cmb(5, 1027, datagen.KINDS + ("ddcfor", "ddc2", "ole", "rle", "sdc")),
    "every kind": lambda: datagen.random_cmb(6, 5003, datagen.KINDS + ("ddcfor", "ddc2", "ole", "rle", "sdc")),
    "next to byte maps": lambda: datagen.random_cmb(7, 5003, ("ddc",) * 20 + ("sdc", "rle", "unc", "ole", "const", "sdcs")),
    "cocoded": lambda: _cocoded(4161),
    "wide dense": lambda: _wide_dense(4127),
    "16-bit maps": lambda: _ddc(17001, [300, 1000, 5000, 257], 3, const=True),
    "mixed kinds side by side": lambda: datagen.random_cmb(9, 70001, ("ddc", "sdcz", "rle", "unc") * 16),
    "a kind per 32 columns": lambda: _by_kind(18817),  # decompress by columns
}


def _plan_bytes(cmb):
    st = native.cla_stats()
    check(native.lib().cla_stats_get(cmb.handle(), st))
    return st.device_bytes


def _use(cmb):
    X = dense_of(cmb)
    for _ in range(2):
        _check(cmb, ks=(1, 2, 5, 9, 65), qs=(1, 3, 9))
        got = np.array(CLALibDecompress.decompress(cmb))
        assert np.array_equal(got, X) or rel_err(got, X, np.abs(X) + 1e-300) < TOL
        got = CLALibTSMM.leftMultByTransposeSelf(cmb)
        assert rel_err(got, X.T @ X, np.abs(X).T @ np.abs(X) + 1e-300) < TOL


@pytest.mark.gpu
@pytest.mark.parametrize("kind", list(BLOCKS))
def test_products_without_room_for_plans(kind):
    cmb = BLOCKS[kind]().to_device()
    before = _plan_bytes(cmb)
    _use(cmb)
    total = _plan_bytes(cmb) - before
    cmb.free()
    assert total > 0
    for limit in sorted({0, total // 8, total // 2, total - 1}):
        cmb = BLOCKS[kind]().to_device()
        check(native.lib().cla_set_plan_limit(cmb.handle(), limit))
        before = _plan_bytes(cmb)
        _use(cmb)
        # (what no kernel does without, a record per column, is not counted)
        assert _plan_bytes(cmb) - before <= limit + 64 * cmb.clen
        cmb.free()


@pytest.mark.gpu
def test_self_product_where_device_memory_is_short():
    """t(X) X in digits can need more scratch than the FP64 products: where only theirs fits, the call works all the same, and
    so does the next one."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(3)
    n, cols = 100_000, 130
    groups = [cg.ColGroupDDC([c], rng.standard_normal((9, 1)), MapToFactory.create_from(rng.integers(0, 9, n), 9)) for c in range(cols)]
    block = CompressedMatrixBlock(n, cols, groups)
    X = torch.from_numpy(dense_of(block)).cuda()
    want, s = (X.T @ X).cpu().numpy(), (X.abs().T @ X.abs()).cpu().numpy()
    del X
    out = torch.empty((cols, cols), dtype=torch.float64, device="cuda")
    lib = native.lib()

    def product(cmb):
        out.zero_()
        rc = lib.cla_tsmm_dev(cmb.handle(), out.data_ptr(), torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        return rc, rel_err(out.cpu().numpy(), want, s + 1e-300)

    for limit in (-1, 0):  # enough memory; both sides' kernels are loaded
        cmb = block.to_device()
        check(lib.cla_set_plan_limit(cmb.handle(), limit))
        rc, err = product(cmb)
        assert rc >= 0 and err < TOL
        cmb.free()
    # scratch of the FP64 products: n x 130 doubles and 16 MiB, 115 MiB; of the digits: planes of 256 columns x 7 bytes, 188
    for left in (130, 150, 180, 260):
        torch.cuda.empty_cache()
        cmb = block.to_device()
        rest = torch.cuda.mem_get_info()[0] - (left << 20)
        hold = [torch.empty(1 << 28, dtype=torch.uint8, device="cuda") for _ in range(rest >> 28)]
        for step in (26, 22):
            while torch.cuda.mem_get_info()[0] - (left << 20) > 1 << step:
                hold.append(torch.empty(1 << step, dtype=torch.uint8, device="cuda"))
        for _ in range(2):
            rc, err = product(cmb)
            assert rc >= 0, (left, native.last_error())
            assert err < TOL, left
        del hold
        cmb.free()


def test_plan_limit_of_an_unknown_handle():
    assert native.lib().cla_set_plan_limit(123456789, 0) == -1
