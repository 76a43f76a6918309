"""The exact second stage of the tensor-core quantizers: lists that are empty, full or over, rows whose norm the tensor-core kernel
cannot take beside rows it can, rows at the codebook's boundaries, one block's tiles and all blocks' -- the packed bytes are
those of the reference-order kernels, and the rows done again are counted."""
import ctypes

import pytest

import project_tensor_b200 as tg
from project_tensor_b200 import _native

pytestmark = pytest.mark.gpu

MODES = ("plain", "all_odd", "some_odd", "first_half_odd", "axes", "zeros", "equal")


def _rows(mode, n, d):
    import torch
    x = torch.randn(n, d, device="cuda", generator=torch.Generator("cuda").manual_seed(n + d))
    if mode == "all_odd":            # sum of squares below 1e-30
        x *= 1e-18
    elif mode == "some_odd":
        x[::37] *= 1e-18
    elif mode == "first_half_odd":
        x[: n // 2] *= 1e-18
    elif mode == "axes":
        x = torch.eye(d, device="cuda")[torch.arange(n, device="cuda") % d] * 3.0
    elif mode == "zeros":
        x[::2] = 0
    elif mode == "equal":
        x = x[:1].expand(n, d).contiguous()
    return x


@pytest.mark.parametrize("kind,d,bits,n", [("prod", 128, 4, 40037), ("mse", 128, 4, 9601), ("prod", 64, 3, 19001), ("mse", 64, 6, 9601),
                                           ("prod", 96, 6, 7233), ("mse", 96, 4, 38000), ("prod", 128, 2, 4737), ("prod", 256, 4, 9601),
                                           ("mse", 256, 2, 4737)])
@pytest.mark.parametrize("mode", MODES)
def test_lists_of_every_length(lib_built, kind, d, bits, n, mode):
    import torch
    quant = (tg.TurboQuantProd if kind == "prod" else tg.TurboQuantMSE)(d, bits, seed=2026, grid_size=4097, max_iter=64)
    x = _rows(mode, n, d)
    packed = {}
    for path in ("auto", "exact"):
        quant.set_kernel_path(path)
        packed[path] = tg.packed_buffers(quant.quantize(x))
        if path == "auto" and d != 256:
            count = ctypes.c_int64(-1)
            dev = torch.device("cuda", 0)
            _native.check(_native.load().tq_plan_last_recheck_rows(quant._plans.handle(dev), torch.cuda.current_stream().cuda_stream, ctypes.byref(count)))
            if mode == "all_odd":
                assert n <= count.value < n + 128 * 148          # whole tiles where a block's list ran over
            if mode == "zeros" and kind == "mse":
                assert count.value == 0
    for name, exact in packed["exact"].items():
        if exact is None:
            continue
        if exact.dtype.is_floating_point:
            # (norms: sums of d squares in another order; residual norms: the residual is down to 1/30 of the unit vector, whose
            # coordinates carry 1.5e-7)
            assert float(((packed["auto"][name] - exact).abs() / exact.abs().clamp_min(1e-37)).max()) <= (6e-7 if name == "norms" else 8e-6), name
        else:
            assert torch.equal(packed["auto"][name], exact), name
