"""The pair transition (px_transition) against fp64 at the edges of its 128-row tiles and of the tiles per CTA: its rows are normalised
eight at a time by eight lanes each, its hidden chunks taken in turn by two groups of warps."""
import pytest
import torch
import torch.nn.functional as F

from protenix_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows", [1, 2, 6, 31, 127, 128, 129, 148 * 128 - 3, 148 * 128 + 1, 300 * 128 + 77])
def test_transition_rows(rows, dtype):
    g = torch.Generator("cuda").manual_seed(rows)
    draw = lambda *s: torch.randn(*s, generator=g, device="cuda")
    x = ((0.5 + draw(rows, 128)) * (0.3 + draw(rows, 1).abs())).to(dtype)
    gamma, beta = 1 + 0.2 * draw(128), 0.2 * draw(128)
    w_a, w_b, w_o = (0.09 * draw(512, 128)).half(), (0.09 * draw(512, 128)).half(), (0.05 * draw(128, 512)).half()
    y = F.layer_norm(x.double(), (128,), gamma.double(), beta.double(), 1e-5)
    update = (F.silu(y @ w_a.double().T) * (y @ w_b.double().T)) @ w_o.double().T
    # operands of 11 bits (normalised rows and hidden values), the result rounded to its own type
    tol = 5e-4 if dtype == torch.float32 else 3e-3
    for residual, in_place in [(False, False), (True, False), (True, True)]:
        src = x.clone()
        out = src if in_place else torch.full_like(x, float("nan"))
        ops.transition(src, out, gamma, beta, w_a, w_b, w_o, residual)
        ops.device_error_flags()
        want = update + x.double() if residual else update
        rel = float((out.double() - want).norm() / want.norm())
        assert rel < tol, (rel, residual, in_place)
