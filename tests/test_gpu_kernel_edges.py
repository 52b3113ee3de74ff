"""Kernels at the edges of their tiles and of the ranges in which each is chosen, against 64-bit restatements."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"


def rnd(*shape, seed, scale=1.0, dtype=torch.float32):
    g = torch.Generator().manual_seed(seed)
    return (torch.randn(*shape, generator=g) * scale).to(dtype).to(DEV)


# ---- short causal convolution ------------------------------------------------------------------------------------------
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("K", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("C, pad", [(516, 0), (20, 12), (18, 0), (640, 1)])
@pytest.mark.parametrize("lens", [[8], [1, 2, 3, 30], [7, 1, 24, 33, 64]])
def test_causal_convolution_over_runs_of_rows(dtype, K, C, pad, lens):
    """Sequences shorter than the filter, ends inside and at the end of a thread's rows, padding rows, channels that are
    and are not whole vectors, rows that lie apart; then the renewed states."""
    from garlic_inference_b200.ops import kernels
    n = sum(lens) + 1
    x = rnd(n, C + pad, seed=1, dtype=dtype)[:, :C]
    taps, bin_, bout = rnd(C, K, seed=2, scale=0.5, dtype=dtype), rnd(C, seed=3), rnd(C, seed=4)
    state = rnd(len(lens) + 2, max(1, K - 1) * C, seed=5)
    order = list(range(len(lens)))[::-1]                                   # slots in another order than the rows
    slots = torch.tensor(sum(([s] * m for s, m in zip(order, lens)), []) + [-1], dtype=torch.int32, device=DEV)
    before = state.clone()
    got = kernels.causal_conv_silu(x, taps, state, slots, activation="silu", in_bias=bin_, out_bias=bout)
    kernels.conv_state_update(x, K, state, slots, in_bias=bin_)
    xd, td, at = x.double() + bin_.double(), taps.double(), 0
    want_state = before.double()
    for s, m in zip(order, lens):
        seen = torch.cat([before[s, :(K - 1) * C].double().view(K - 1, C), xd[at:at + m]])
        z = bout.double() + sum(seen[j:j + m] * td[:, j] for j in range(K))
        mag = bout.double().abs() + sum((seen[j:j + m] * td[:, j]).abs() for j in range(K))
        # K + 1 roundings of the sum and of the biased input (silu's slope stays below 1.1), then silu's own
        tol = 1.1 * (2 * K + 2) * 2.0 ** -24 * mag + 2.0 ** -20 * z.abs()
        assert ((got[at:at + m].double() - z * torch.sigmoid(z)).abs() <= tol + 1e-7).all()
        if K > 1:
            want_state[s, :(K - 1) * C] = seen[m:].reshape(-1)
        at += m
    assert (state.double() - want_state).abs().max() <= 2.0 ** -23 * 8
