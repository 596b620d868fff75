"""The per-token products' input, assembled by all threads of a block, and their outputs in windows of rows, against float64.

Bars: a product sums cols fp32 terms in fixed trees of at most 2^13 terms a thread and warp, a few units of 2^-24 of the terms' magnitude; norms add the same."""
import ctypes as C

import numpy as np
import pytest

import _latent as T

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
Q8, F16 = 0, 1


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).cuda()


def packed(lib, w, wtype):
    """Rows as the kernel reads them and the values they hold."""
    rows, cols = w.shape
    stride = lib.b200_packed_row_stride(wtype, cols)
    d, src = torch.zeros(rows, stride, dtype=torch.uint8, device="cuda"), dev(w)
    call = lib.b200_q8_pack if wtype == Q8 else lib.b200_f16_pack
    assert call(src.data_ptr(), cols, rows, cols, d.data_ptr(), stride, 0, 1, None) == 0
    torch.cuda.synchronize()
    if wtype == F16:
        return d, stride, src.half().double()
    raw = d.cpu().numpy()
    quants = raw[:, :cols].view(np.int8).astype(np.float64)
    scales = np.ascontiguousarray(raw[:, cols:cols + cols // 16]).view(np.float16).astype(np.float64)
    return d, stride, torch.from_numpy(quants * np.repeat(scales, 32, axis=1)).cuda()


def resid_call(lib, pkg, d, stride, rows, cols, wtype, resid, slots, norm_at, final, grid=0):
    a = pkg.MatvecArgs()
    a.d_w, a.row_stride, a.rows, a.cols, a.wtype, a.in_mode, a.out_mode, a.n_out, a.eps, a.grid = d.data_ptr(), stride, rows, cols, wtype, pkg.B200_IN_RESID, \
        pkg.B200_OUT_STORE, 1, 1e-5, grid
    out, kept = torch.full((rows,), float("nan"), device="cuda"), torch.full((cols,), float("nan"), device="cuda")
    a.d_out[0], a.d_resid_in, a.d_resid_out, a.n_slots, a.slot_stride = out.data_ptr(), resid.data_ptr(), kept.data_ptr(), len(slots), cols
    a.d_slots = slots.data_ptr() if len(slots) else None
    a.d_slot_norm_gamma = norm_at
    a.d_norm_gamma = final.data_ptr() if final is not None else None
    assert lib.b200_matvec(C.byref(a), None) == 0
    torch.cuda.synchronize()
    return out, kept


@pytest.mark.parametrize("wtype", [Q8, F16])
@pytest.mark.parametrize("cols", [32, 512, 2560, 4096, 5120, 9728])
@pytest.mark.parametrize("grid", [0, 3])
def test_slot_norm_weights_on_any_element(lib, pkg, wtype, cols, grid):
    """The weights of the slots' norm one to three elements behind a 16-byte boundary: the same bits."""
    g = torch.Generator().manual_seed(cols)
    w = torch.randn(37, cols, generator=g).numpy()
    d, stride, _ = packed(lib, w, wtype)
    resid, slots, gamma = torch.randn(cols, generator=g).cuda(), torch.randn(2, cols, generator=g).cuda(), torch.randn(cols, generator=g)
    got = []
    for off in range(4):
        room = torch.full((cols + 8,), float("nan"))
        room[off:off + cols] = gamma
        room = room.cuda()
        assert room.data_ptr() % 16 == 0
        got.append(resid_call(lib, pkg, d, stride, 37, cols, wtype, resid, slots, room.data_ptr() + 4 * off, None, grid))
    for out, kept in got:
        assert not torch.isnan(out).any() and torch.equal(out, got[0][0]) and torch.equal(kept, got[0][1])
