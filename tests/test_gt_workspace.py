"""Device memory of the tensor kNN: what the staged scan asks for, computed by the engine's own layout code on the
host (nbpg_test_gt_workspace), against the replaying engine that ran these calls before it."""
import ctypes as C
import itertools
import os


def _sizes(dtype, dims, n, nq, k, sms=152):
    from nbpg_gb300 import _lib, build_ext
    if not os.path.exists(_lib.LIB_PATH):
        build_ext.build()
    scan, replay = C.c_size_t(), C.c_size_t()
    _lib.check(_lib.lib().nbpg_test_gt_workspace(_lib.DTYPES[dtype], dims, n, nq, k, sms, C.byref(scan), C.byref(replay)))
    return scan.value, replay.value


def test_scan_needs_no_more_than_the_replaying_engine():
    """Rows of up to 128 codes and k <= 100 ran on the replaying engine: a call that had room for it has room
    for the staged scan.  (Shorter bases, for which the replaying engine has few ranges, may take up to 128 MB more; a
    call without that much still goes on to the replaying engine.)"""
    for n, nq, k, (dtype, dims), sms in itertools.product(
            (1000, 5000, 50003, 200000, 1000000, 100000000), (1, 17, 128, 129, 300, 2048, 10000, 16384, 16385, 100000),
            (1, 10, 16, 25, 26, 32, 48, 51, 52, 64, 100), (("u8", 128), ("u4", 32), ("i8", 1)), (148, 152)):
        if k > n:
            continue
        scan, replay = _sizes(dtype, dims, n, nq, k, sms)
        assert scan <= replay + (0 if n >= 1000000 else 128 << 20), (n, nq, k, dtype, dims, sms, scan, replay)


def test_one_query_takes_megabytes():
    """Lists are kept for the queries there are: one query over 1M rows needs the bf16 copy of the base and a few MB."""
    for k in (1, 10, 100, 128):
        scan, _ = _sizes("u8", 128, 1000000, 1, k)
        assert scan - 1000064 * (256 + 4) < 8 << 20, (k, scan)
