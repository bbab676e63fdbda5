"""The workspace queries cover every layout that the calls behind them may choose."""
import pytest
import torch

from flaggems_b200 import _cabi


@pytest.mark.skipif(torch.cuda.is_available(), reason="passes made-up addresses: for hosts where nothing can be launched")
def test_grouped_mm_workspace_covers_the_call():
    lib = _cabi.lib()
    for groups in (1, 3, 8, 32, 256, 1024):
        for per_group in (1, 31, 33, 127, 500, 767, 768, 1000, 4096, 20000, 33000, 40000, 65536, 262144):
            for m in (groups * per_group, groups * per_group + 1, groups * per_group - 1):
                if not 0 < m < (1 << 28):
                    continue
                need = lib.fg_scaled_grouped_mm_workspace_bytes(m, groups, 128)
                for n in (16, 128, 240, 256, 4096, 7168):
                    rc = lib.fg_scaled_grouped_mm_fp8(4096, 4096, 4096, 4096, 4096, None, 0, 4096, groups, m, n, 128, 128, n, 0,
                                                      4096, need, None)
                    text = lib.fg_last_error().decode()
                    assert rc != 0 and "workspace" not in text, (groups, m, n, text)


@pytest.mark.skipif(torch.cuda.is_available(), reason="as above")
def test_grouped_mm_workspace_one_byte_short_is_refused():
    lib = _cabi.lib()
    need = lib.fg_scaled_grouped_mm_workspace_bytes(100, 2, 128)
    rc = lib.fg_scaled_grouped_mm_fp8(4096, 4096, 4096, 4096, 4096, None, 0, 4096, 2, 100, 64, 128, 128, 64, 0, 4096, need - 1, None)
    assert rc == -1 and "workspace holds" in lib.fg_last_error().decode()
