"""The C ABI without a GPU: the library builds, loads, and exports every symbol include/niti_b200.h declares."""
import ctypes
import os
import re

from tests.conftest import ROOT


def declared_symbols():
    text = open(os.path.join(ROOT, "include", "niti_b200.h")).read()
    return sorted(set(re.findall(r"NITI_API\s+[\w\s\*]+?\b(niti_\w+)\s*\(", text)))


def test_library_builds_and_exports_every_declared_symbol():
    from niti_b200 import build
    lib = ctypes.CDLL(build.build())
    names = declared_symbols()
    assert len(names) >= 20
    for n in names:
        assert hasattr(lib, n), f"{n} is declared in include/niti_b200.h but not exported"


def test_ctypes_table_matches_header():
    from niti_b200 import _lib
    assert sorted(_lib.SIGNATURES) == declared_symbols()


def test_error_strings_and_argument_checks_need_no_gpu():
    from niti_b200 import _lib
    L = _lib.lib
    assert L.niti_version() >= 100
    assert L.niti_strerror(0) == b"ok"
    for code in (-1, -2, -3, -4):
        assert len(L.niti_strerror(code)) > 5
    # null pointers / bad sizes are rejected before any CUDA call
    assert L.niti_requant_i8(None, None, None, 16, 0, 7, 0, None, 0, 0, 0, None, None, None, None, None) == -1
    assert L.niti_conv_fprop_i8(None, None, None, None, None, 0, 1, 8, 8, 128, 128, 3, 3, 1, 1, None, None) == -1
    assert L.niti_conv_wgrad_scratch_bytes(0, 8, 8, 128, 128, 3, 3) == 0
    assert L.niti_conv_fprop_requant_supported(128, 128, 3, 3, 1) == 1
    assert L.niti_conv_fprop_requant_supported(100, 128, 3, 3, 1) == 0


def test_front_end_is_rebuilt_for_another_torch(monkeypatch):
    from niti_b200 import build
    build.build()
    assert not build.ops_stale()
    monkeypatch.setattr(build.metadata, "version", lambda name: "99.0")  # as after an upgrade of torch
    assert build.ops_stale()


def test_entry_points_without_scratch_follow_the_reduction_switch():
    from niti_b200._lib import lib
    assert lib.niti_conv_wgrad_update_elems(16, 16, 3, 3, 1) > 0 and lib.niti_conv_wgrad_batch_inner_supported(16, 16, 16, 3, 3, 1) == 1
    old = lib.niti_set_option(2, 0)
    try:
        assert lib.niti_conv_wgrad_update_elems(16, 16, 3, 3, 1) == 0 and lib.niti_conv_wgrad_batch_inner_supported(16, 16, 16, 3, 3, 1) == 0
    finally:
        lib.niti_set_option(2, old)


def test_padded_products_leave_deep_reductions_with_few_results_to_the_cuda_cores():
    from niti_b200._lib import lib
    padded = lambda *a: lib.niti_gemm_scratch_bytes(*a) > 0
    for M, N, K in [(1, 2048, 8192), (10, 259, 8032), (61, 112, 5472), (498, 24, 8064), (2, 4096, 4096)]:
        assert not padded(M, N, K, 0, 1)
    assert padded(245, 127, 640, 0, 1) and padded(18, 112, 8886, 1, 0) and padded(607, 48, 725, 0, 0)
    assert not padded(929, 544, 54, 1, 0) and padded(1020, 400, 143, 1, 0)


def test_the_reference_arm_without_the_reference_says_so():
    import json
    import subprocess
    import sys
    import pytest
    if os.path.isfile(os.path.join(ROOT, "oracle", "_ref", "ti_torch.py")):
        pytest.skip("the reference's Python is here")
    out = subprocess.run([sys.executable, os.path.join(ROOT, "bench.py"), "--impl", "reference"], capture_output=True, text=True, timeout=300, check=True)
    line = json.loads(out.stdout.strip().splitlines()[-1])
    assert line["impl"] == "reference" and line["unavailable"] and "value" not in line


def test_dealing_thread_blocks_to_layers_is_no_work_for_the_host():
    """Weight gradients whose items are more than the SMs are dealt by simulated schedules in every call that is not captured: within a
    few times the call's other host work (a schedule block by block was 25 to 60 times).  Without a GPU the call ends
    behind the deal with an error; its addresses are never used."""
    import time

    import pytest
    import torch
    from niti_b200._lib import WgradItem, lib
    if torch.cuda.is_available():
        pytest.skip("would launch on addresses that are none")

    def least(shapes):
        items = (WgradItem * len(shapes))(*[WgradItem(1 << 20, 1 << 21, 1 << 22, *s, 3, 3, 1) for s in shapes])
        best = 1.0
        for _ in range(500):
            t = time.perf_counter()
            assert lib.niti_conv_wgrad_accumulate_multi_i8(items, len(shapes), None, None) == -3
            best = min(best, time.perf_counter() - t)
        return best
    plain = least([(128, 8, 8, 512, 512), (128, 8, 8, 256, 512)])
    for shapes in ([(1024, 4, 4, 512, 512), (1024, 4, 4, 512, 512), (1024, 8, 8, 512, 512), (1024, 8, 8, 256, 512)],
                   [(2, 4, 4, 1024, 1024), (16, 8, 8, 512, 512)]):
        assert least(shapes) < 15 * plain
