"""aether_conv2d_act_fwd with every row length and alignment of the operand copy that it accepts, on the kernels that write the
activation in their epilogue (per-tap) and on those that leave it to a pass behind (window kernel, CTA pairs, TF32): the
activation is that of the layer's output and the copy its bf16 rounding, bit for bit, zero in the padded columns, and
nothing beside the copy is written."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu

#          S, H, W, Cin, Cout, f, mode
SHAPES = [(7, 1, 1, 64, 36, 1, "bf16"), (130, 1, 1, 100, 64, 1, "bf16"), (40000, 1, 1, 64, 100, 1, "bf16"), (2, 56, 56, 16, 20, 3, "bf16"),
          (33, 1, 1, 48, 36, 1, "tf32"), (3, 9, 8, 32, 100, 3, "tf32")]


@pytest.mark.parametrize("S,H,W,Cin,Cout,f,mode", SHAPES)
def test_copy_rows(S, H, W, Cin, Cout, f, mode):
    import torch
    from aether_ml_b200 import _lib
    L = _lib.lib()
    d = _lib.AetherConvDesc(S, H, W, Cin, Cout, f, f, 1, 1, (f - 1) // 2, (f - 1) // 2, _lib.MATH_MODES[mode])
    g = torch.Generator(device="cuda").manual_seed(S)
    x, w = torch.randn((S, H, W, Cin), generator=g, device="cuda"), torch.randn((f, f, Cin, Cout), generator=g, device="cuda")
    b = torch.randn(Cout, generator=g, device="cuda")
    rows = S * H * W
    y, act = torch.empty((rows, Cout), device="cuda"), torch.empty((rows, Cout), device="cuda")
    ws = torch.empty(L.aether_conv2d_workspace_bytes(C.byref(d)), dtype=torch.uint8, device="cuda")
    p = lambda t: C.c_void_p(t.data_ptr())
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    padded = (Cout + 63) // 64 * 64
    for ld in sorted({Cout, min(Cout + 4, padded), padded}):
        for shift in (0, 4):                                  # a base of 16-byte and of 8-byte alignment
            room = torch.full((rows * ld + 64,), 7.0, dtype=torch.bfloat16, device="cuda")
            rc = L.aether_conv2d_act_fwd(C.byref(d), p(x), p(w), p(b), p(y), p(act), 0.125, C.c_void_p(room.data_ptr() + 2 * (16 + shift)), ld,
                                         p(ws), ws.numel(), 0, st)
            assert rc == 0, L.aether_last_error()
            assert torch.equal(act, torch.where(y > 0, y, y * 0.125))
            copy = room[16 + shift:16 + shift + rows * ld].view(rows, ld)
            assert torch.equal(copy[:, :Cout], act.bfloat16()) and bool((copy[:, Cout:] == 0).all()), (ld, shift)
            assert bool((room[:16 + shift] == 7).all()) and bool((room[16 + shift + rows * ld:] == 7).all()), (ld, shift)
    for ld, base in ((Cout + 2, 0), (Cout - 4, 0), (padded + 4, 0), (Cout, 2)):       # refused before anything is launched
        n = _lib.launch_count()
        rc = L.aether_conv2d_act_fwd(C.byref(d), p(x), p(w), p(b), p(y), p(act), 0.125, C.c_void_p(room.data_ptr() + 2 * base), ld, p(ws),
                                     ws.numel(), 0, st)
        assert rc != 0 and _lib.launch_count() == n, (ld, base)
    assert _lib.device_status() == 0
