"""Which width of the whole-token kernel a plan takes, and that its geometry keeps to it (no GPU)."""
import ctypes as C

import pytest

from test_cpu_token_plan import planned


@pytest.mark.parametrize("arch,tp,wtype,consumers", [("tiny-qwen3", 1, 0, 320), ("tiny-qwen3", 1, 1, 320), ("tiny-gemma3", 1, 0, 320), ("tiny-qwen3", 2, 0, 640),
                                                     ("qwen3-4b", 1, 0, 640), ("gemma3-1b", 1, 1, 640)])
def test_width(lib, pkg, arch, tp, wtype, consumers):
    rc, a = planned(lib, pkg, arch, wtype, tp)
    assert rc == 0 and a.consumers == consumers
    for g in a.g:
        assert g.T * g.NG <= consumers and g.T * g.spt * (8 if wtype else 16) >= g.cols
        assert consumers == 640 or g.spt == 1


def test_groups_of_eight_stay_wide(lib, pkg):
    rc, a = planned(lib, pkg, "tiny-qwen3", 0, 1)
    assert rc == 0 and a.consumers == 320
    b = pkg.TokenArgs.from_buffer_copy(a)
    b.n_q, b.n_kv = 8, 1
    b.g[0].rows = 10 * b.hd
    assert lib.b200_token_plan(C.byref(b), 148) == 0 and b.consumers == 640
