"""Complex64 K / K^H where the coefficient-row kernel's tiles are ragged: rows
shorter and longer than 32 nodes, fewer rows than a CTA holds, every batch size.

Against the complex128 rows: six products per node, coefficients and values
rounded to fp32 (6e-8 each), so 2e-6 is far above the error of a right row and
far below that of a wrong neighbour or coefficient."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(31, 7, 3), (32, 8, 2), (33, 9, 4), (70, 3, 5), (5, 17, 2)])
@pytest.mark.parametrize("nrhs", [1, 2, 3, 4, 5, 8])
def test_coefficient_rows(shape, nrhs):
    from ultrasound_solver_b200 import _native as N
    from ultrasound_solver_b200.scene import DeviceOperator
    gen = torch.Generator(device="cuda").manual_seed(nrhs)
    n = int(np.prod(shape))
    rand = lambda: torch.rand(n, dtype=torch.float64, device="cuda", generator=gen)
    op = DeviceOperator(shape, 1e-3, 2 * np.pi * 4e4,
                        {"-x": "open", "+x": "soft", "-y": "soft", "+z": "open"}, 1.2 * (1 + 0.3 * rand()),
                        343 * (1 + 0.1 * rand()))
    x = torch.randn((nrhs, n), dtype=torch.complex64, device="cuda", generator=gen)
    for variant in (N.APPLY_K, N.APPLY_KH):
        got = op.apply(x, variant, N.PREC_MIXED, kernel=N.STENCIL_COEF_ROWS).to(torch.complex128)
        want = op.apply(x.to(torch.complex128), variant, N.PREC_FP64)
        err = torch.linalg.norm(got - want, dim=1) / torch.linalg.norm(want, dim=1)
        assert float(err.max()) < 2e-6


@pytest.mark.parametrize("shape", [(33, 257, 250), (70, 129, 121), (97, 90, 83)])
def test_bulk_copied_rows(shape):
    """Operands beyond the L2 (93 MB): coefficients by bulk copies, ragged in x
    and y, against the complex128 rows (bound as above), and bit for bit the
    right-hand sides one at a time (smaller operands, read directly where the
    grid is the last one's)."""
    from ultrasound_solver_b200 import _native as N
    from ultrasound_solver_b200.scene import DeviceOperator
    gen = torch.Generator(device="cuda").manual_seed(3)
    n = int(np.prod(shape))
    rand = lambda: torch.rand(n, dtype=torch.float64, device="cuda", generator=gen)
    op = DeviceOperator(shape, 1e-3, 2 * np.pi * 4e4,
                        {"-x": "open", "+x": "soft", "-y": "soft", "+z": "open"}, 1.2 * (1 + 0.3 * rand()),
                        343 * (1 + 0.1 * rand()))
    x = torch.randn((8, n), dtype=torch.complex64, device="cuda", generator=gen)
    for variant in (N.APPLY_K, N.APPLY_KH):
        want = op.apply(x.to(torch.complex128), variant, N.PREC_FP64)
        one = torch.stack([op.apply(v, variant, N.PREC_MIXED, kernel=N.STENCIL_COEF_ROWS) for v in x])
        for nrhs in (2, 3, 4, 5, 8):
            got = op.apply(x[:nrhs].contiguous(), variant, N.PREC_MIXED, kernel=N.STENCIL_COEF_ROWS)
            assert torch.equal(got, one[:nrhs])
            err = torch.linalg.norm(got.to(torch.complex128) - want[:nrhs], dim=1)
            assert float((err / torch.linalg.norm(want[:nrhs], dim=1)).max()) < 2e-6
