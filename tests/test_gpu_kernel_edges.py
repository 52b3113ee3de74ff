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


# ---- gates of the recurrent unit -------------------------------------------------------------------------------------------
@pytest.mark.parametrize("blocks, bw", [(3, 8), (2, 64), (3, 72), (2, 320), (2, 20)])
@pytest.mark.parametrize("n", [1, 17, 128, 129, 300])
def test_recurrent_gates_with_bfloat16_matrices(blocks, bw, n):
    """Blocks narrower than a tile of outputs, whole and part tiles of outputs, inputs and rows; an infinite input; the
    same bits for a row alone and among others."""
    from garlic_inference_b200.ops import kernels
    W = blocks * bw
    u = rnd(n, W, seed=1, scale=2.0)
    u[n - 1, 1] = math.inf
    wa, wi = (rnd(blocks, bw, bw, seed=s, scale=bw ** -0.5, dtype=torch.bfloat16) for s in (2, 3))
    ba, bi, lam = rnd(W, seed=4), rnd(W, seed=5), rnd(W, seed=6, scale=2.0)
    a, b = kernels.rglru_gates(u, wa, wi, ba, bi, lam, 8.0)
    ud = u.double().view(n, blocks, bw)
    z = [torch.einsum("nbi,bio->nbo", ud, w.double()).reshape(n, W) + v.double() for w, v in ((wa, ba), (wi, bi))]
    # every addition of a partial sum may lose one unit of the largest partial sum's last place
    dz = [(3 * bw / 16 + 3) * 2.0 ** -23 * (torch.einsum("nbi,bio->nbo", ud.abs(), w.double().abs()).reshape(n, W) + v.double().abs())
          for w, v in ((wa, ba), (wi, bi))]
    log_a = -8.0 * torch.sigmoid(z[0]) * torch.nn.functional.softplus(lam.double())
    want_a = torch.exp(log_a)
    want_b = torch.sqrt(-torch.expm1(2 * log_a)) * torch.sigmoid(z[1]) * u.double()
    fine = torch.ones(n, W, dtype=torch.bool, device=DEV)
    fine[n - 1, :bw] = False                                               # the block that holds the infinite input
    tol_a = want_a * (log_a.abs() * (dz[0] + 2.0 ** -20) + 2.0 ** -21)
    tol_b = want_b.abs() * (dz[0] + dz[1] + 2.0 ** -19)
    assert ((a.double() - want_a).abs() <= tol_a + 1e-30)[fine].all()
    assert ((b.double() - want_b).abs() <= tol_b + 1e-30)[fine].all()
    torch.testing.assert_close(a[n - 1, :bw].double(), want_a[n - 1, :bw], rtol=1e-5, atol=1e-30)
    assert torch.equal(b[n - 1, :bw].isfinite(), want_b[n - 1, :bw].isfinite())
    alone = kernels.rglru_gates(u[n // 2:n // 2 + 1].contiguous(), wa, wi, ba, bi, lam, 8.0)
    assert torch.equal(alone[0][0], a[n // 2]) or bool(alone[0][0].isnan().any())


# ---- scan of the recurrent unit --------------------------------------------------------------------------------------------
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("width, pad", [(32, 8), (100, 0), (66, 2), (35, 0), (324, 4)])
@pytest.mark.parametrize("lens", [[1, 2], [3, 4, 5], [59, 60, 61], [64, 130, 1]])
def test_recurrent_scan_at_the_ends_of_its_ring(dtype, width, pad, lens):
    """Sequences around the number of tokens that are under way, channels that are and are not whole warps and whole
    16-byte words, and a portion of padding rows."""
    from garlic_inference_b200.ops import kernels
    n = sum(lens) + 3
    a, b = torch.rand(n, width, generator=torch.Generator().manual_seed(1)).to(DEV), rnd(n, width, seed=2)
    y, yb, state = rnd(n, width + pad, seed=3, dtype=dtype)[:, :width], rnd(width, seed=4), rnd(len(lens) + 1, width + 4, seed=5)
    starts = [sum(lens[:i]) for i in range(len(lens))]
    spans = torch.tensor([[i, s, m] for i, (s, m) in enumerate(zip(starts, lens))] + [[-1, n - 3, 3]], dtype=torch.int32, device=DEV)
    before, slots = state.clone(), torch.zeros(n, dtype=torch.int32, device=DEV)
    got = kernels.rglru_scan(a, b, y, yb, state, spans, slots)
    act = torch.nn.functional.gelu(y.double() + yb.double(), approximate="tanh")
    for i, (s, m) in enumerate(zip(starts, lens)):
        S, low = before[i, :width].double(), torch.zeros(width, dtype=torch.float64, device=DEV)
        for t in range(s, s + m):
            S = a[t].double() * S + b[t].double()
            low = a[t].double() * low + 2.0 ** -23 * S.abs()               # a rounding a token, carried along
            tol = (low + 1e-6) * act[t].abs() + (2.0 ** -20 if dtype == torch.float32 else 2.0 ** -7) * (S * act[t]).abs() + 1e-6
            if dtype == torch.bfloat16:                                    # the hardware's tanh: 2^-10.9 of 1
                tol = tol + 0.5 * 2.0 ** -10 * (S * (y[t].double() + yb.double())).abs()
            assert ((got[t].double() - S * act[t]).abs() <= tol).all()
        assert ((state[i, :width].double() - S).abs() <= low + 1e-6).all()
    assert float(got[n - 3:].abs().max()) == 0.0 and torch.equal(state[len(lens)], before[len(lens)])
    assert torch.equal(state[:, width:], before[:, width:])


# ---- float32 product -------------------------------------------------------------------------------------------------------
@pytest.mark.parametrize("N, K", [(1, 4), (17, 7), (64, 128), (200, 130), (1100, 260), (4800, 36)])
def test_float32_product_has_the_same_bits_by_every_kernel(N, K):
    """Row counts on both sides of every choice of kernel and tile, sizes that are and are not whole tiles, slices and
    16-byte words, rows that lie apart: all against 64 bits, and every row with the bits of its product alone."""
    from garlic_inference_b200.ops import kernels
    w, full = rnd(N, K, seed=1), rnd(700, K + 5, seed=2)
    alone = {}
    for M in (1, 3, 4, 5, 8, 9, 16, 17, 32, 33, 64, 65, 129, 300, 700):
        for a in (full[:M, :K].contiguous(), full[:M, :K]):
            out = torch.full((M, N + 3), 7.0, device=DEV)
            kernels.sgemm_nt_strided(a, w, out[:, :N])
            want = a.double() @ w.double().T
            tol = (K + 1) * 2.0 ** -24 * (a.double().abs() @ w.double().abs().T)       # a rounding an addition
            assert ((out[:, :N].double() - want).abs() <= tol).all() and bool((out[:, N:] == 7.0).all())
            for r in {0, M // 2, M - 1}:
                one = alone.setdefault(r, kernels.sgemm_nt(full[r:r + 1, :K].contiguous(), w)[0])
                assert torch.equal(out[r, :N], one), f"{M} rows, row {r}"
