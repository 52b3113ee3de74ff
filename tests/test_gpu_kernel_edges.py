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


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("K", [1, 2, 3, 4])
def test_causal_convolution_of_many_elements_has_the_bits_of_few(dtype, K):
    """Rows by the kernel that keeps runs of them, the same columns a few at a time by the kernel of a thread per element."""
    from garlic_inference_b200.ops import kernels
    C, lens = 6152, [7, 1, 24, 33, 64]
    n = sum(lens) + 1
    assert n * C > 3 << 18 > n * 1024
    x, taps, bin_, bout = rnd(n, C, seed=1, dtype=dtype), rnd(C, K, seed=2, dtype=dtype), rnd(C, seed=3), rnd(C, seed=4)
    state = rnd(len(lens), max(1, K - 1) * C, seed=5)
    slots = torch.tensor(sum(([i] * m for i, m in enumerate(lens)), []) + [-1], dtype=torch.int32, device=DEV)
    got = kernels.causal_conv_silu(x, taps, state, slots, in_bias=bin_, out_bias=bout)
    for at in range(0, C, 1024):
        cut = slice(at, min(C, at + 1024))
        w = min(C, at + 1024) - at
        part = state[:, :(K - 1) * C].view(len(lens), K - 1, C)[:, :, cut].reshape(len(lens), -1) if K > 1 else state[:, :w]
        want = kernels.causal_conv_silu(x[:, cut], taps[cut].contiguous(), part.contiguous(), slots, in_bias=bin_[cut].contiguous(),
                                        out_bias=bout[cut].contiguous())
        assert torch.equal(got[:, cut], want)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("K", [2, 3, 4, 6])
@pytest.mark.parametrize("lens", [[1] * 33 + [20], [2] * 300, [1, 2, 3, 4, 5] * 9 + [1] * 500])
def test_convolution_states_of_many_sequences(dtype, K, lens):
    """Steps in which many of neighbouring rows are the last of their sequences, few and many rows, with padding between."""
    from garlic_inference_b200.ops import kernels
    C, rows = 300, []
    order = torch.randperm(len(lens), generator=torch.Generator().manual_seed(1)).tolist()
    for i, m in zip(order, lens):
        rows += [i] * m + ([-1] if i % 7 == 0 else [])
    x, bias, state = rnd(len(rows), C, seed=2, dtype=dtype), rnd(C, seed=3), rnd(len(lens) + 1, (K - 1) * C + 4, seed=4)
    want = state.clone()
    for i in order:
        mine = [r for r, s in enumerate(rows) if s == i]
        seen = torch.cat([state[i, :(K - 1) * C].view(K - 1, C), x[mine].float() + bias])
        want[i, :(K - 1) * C] = seen[len(mine):].reshape(-1)
    kernels.conv_state_update(x, K, state, torch.tensor(rows, dtype=torch.int32, device=DEV), in_bias=bias)
    assert torch.equal(state, want)


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
@pytest.mark.parametrize("blocks, bw", [(64, 64), (16, 320), (4, 1280)])
@pytest.mark.parametrize("scale, shift", [(1.0, 0.0), (0.1, 0.0), (3.0, 0.0), (1.0, 1.0)])
def test_recurrent_gates_on_tensor_cores_are_as_close_as_by_multiply_adds(blocks, bw, scale, shift):
    """The same bfloat16 matrices, given as such (tensor cores) and widened to float32 (multiply-adds): the former is no further
    from 64 bits, in the 2-norm over a million numbers (one part in 100 for the sample)."""
    from garlic_inference_b200.ops import kernels
    W, n = blocks * bw, 256
    u = rnd(n, W, seed=1, scale=scale) + shift
    wa, wi = (rnd(blocks, bw, bw, seed=s, scale=bw ** -0.5, dtype=torch.bfloat16) for s in (2, 3))
    ba, bi = rnd(W, seed=4, scale=0.1), rnd(W, seed=5, scale=0.1)
    keep = 0.9 + 0.099 * torch.rand(W, generator=torch.Generator().manual_seed(6))
    lam = torch.log(torch.expm1(-torch.log(keep) / 8.0)).to(DEV)
    z = [torch.einsum("nbi,bio->nbo", u.double().view(n, blocks, bw), w.double()).reshape(n, W) + b.double()
         for w, b in ((wa, ba), (wi, bi))]
    log_a = -8.0 * torch.sigmoid(z[0]) * torch.nn.functional.softplus(lam.double())
    want = torch.exp(log_a), torch.sqrt(-torch.expm1(2 * log_a)) * torch.sigmoid(z[1]) * u.double()
    tensor, plain = (kernels.rglru_gates(u, wa.to(t), wi.to(t), ba, bi, lam, 8.0) for t in (torch.bfloat16, torch.float32))
    for got, other, w in zip(tensor, plain, want):
        assert (got.double() - w).norm() <= 1.01 * (other.double() - w).norm()


@pytest.mark.parametrize("n", [1, 17, 200])
def test_recurrent_gates_beyond_the_finite_are_those_of_multiply_adds(n):
    """Infinite weights times inputs whose second and third parts are zero, infinite inputs times weights that are and are not
    zero, a NaN whose upper 16 bits are an infinity's: infinities and NaN where the multiply-adds have them."""
    from garlic_inference_b200.ops import kernels
    blocks, bw = 2, 72
    u = rnd(n, blocks * bw, seed=1)
    u[:, 3] = 1.5                                                          # one part
    u[0, 4] = math.inf
    u[n - 1, 80:81].view(torch.int32)[0] = 0x7f800001
    wa, wi = (rnd(blocks, bw, bw, seed=s, scale=bw ** -0.5, dtype=torch.bfloat16) for s in (2, 3))
    wa[0, 3, 5], wa[0, 3, 6], wi[0, 3, 7], wi[0, 4, 8], wa[1, 9, 1] = math.inf, -math.inf, math.inf, 0.0, math.nan
    ba, bi, lam = rnd(blocks * bw, seed=4), rnd(blocks * bw, seed=5), rnd(blocks * bw, seed=6)
    tensor, plain = (kernels.rglru_gates(u, wa.to(t), wi.to(t), ba, bi, lam, 8.0) for t in (torch.bfloat16, torch.float32))
    for got, want in zip(tensor, plain):
        assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isinf(), want.isinf())
        ok = want.isfinite()
        torch.testing.assert_close(got[ok], want[ok], rtol=1e-5, atol=1e-5)
    assert float(tensor[0][n - 1, 6]) == 1.0 or n == 1                     # a gate shut by minus infinity keeps the state


@pytest.mark.parametrize("blocks, bw", [(3, 8), (2, 64), (3, 72), (2, 320), (1, 600)])
@pytest.mark.parametrize("n", [1, 128, 300])
def test_recurrent_gates_of_many_rows(blocks, bw, n, monkeypatch):
    """The tcgen05 kernel: blocks narrower than a tile of outputs, part tiles of outputs, inputs and rows; gates wide open, shut and in
    between, inputs, weights and biases beyond the finite: no further from 64 bits than mma.sync (one part in 50 for the sample), and
    infinities and NaN where that has them."""
    from garlic_inference_b200.ops import kernels
    monkeypatch.setattr(kernels, "_gates_on_tcgen05", lambda n, bw: True)
    W = blocks * bw
    u = rnd(n, W, seed=1, scale=2.0)
    wa, wi = (rnd(blocks, bw, bw, seed=s, scale=bw ** -0.5, dtype=torch.bfloat16) for s in (2, 3))
    wa_t, wi_t = wa.transpose(1, 2).contiguous(), wi.transpose(1, 2).contiguous()
    ba, bi, lam = rnd(W, seed=4), rnd(W, seed=5), rnd(W, seed=6, scale=2.0)
    ba[1], ba[2], bi[1], bi[2], lam[3], lam[4] = 60.0, -120.0, -120.0, 60.0, -30.0, 30.0
    old = kernels.rglru_gates(u, wa_t, wi_t, ba, bi, lam, 8.0)
    new = kernels.rglru_gates(u, wa_t, wi_t, ba, bi, lam, 8.0, wa=wa, wi=wi)
    z = [torch.einsum("nbi,boi->nbo", u.double().view(n, blocks, bw), w.double()).reshape(n, W) + v.double() for w, v in ((wa, ba), (wi, bi))]
    log_a = -8.0 * torch.sigmoid(z[0]) * torch.nn.functional.softplus(lam.double())
    want = torch.exp(log_a), torch.sqrt(-torch.expm1(2 * log_a)) * torch.sigmoid(z[1]) * u.double()
    # one against the other: a = exp(log a) with -log a up to 70 above atol, which magnifies the error of its gate, bw sums that may each
    # lose 2^-24 of it: 70 sqrt(bw) 2^-24 or less, 1e-4
    tol = dict(rtol=70 * bw ** 0.5 * 2.0 ** -24, atol=1e-30)
    for got, other, w in zip(new, old, want):
        assert (got.double() - w).norm() <= 1.02 * (other.double() - w).norm() + 2.0 ** -25 * w.norm()
        torch.testing.assert_close(got, other, **tol)
    u[0, 0], u[n // 2, W - 1], ba[5], bi[6] = math.inf, math.nan, math.inf, -math.inf
    wa[0, 2, 3], wi[blocks - 1, 4, 1] = math.inf, -math.inf
    wa_t, wi_t = wa.transpose(1, 2).contiguous(), wi.transpose(1, 2).contiguous()
    old = kernels.rglru_gates(u, wa_t, wi_t, ba, bi, lam, 8.0)
    for got, other in zip(kernels.rglru_gates(u, wa_t, wi_t, ba, bi, lam, 8.0, wa=wa, wi=wi), old):
        assert torch.equal(got.isnan(), other.isnan()) and torch.equal(got.isinf(), other.isinf())
        torch.testing.assert_close(got[other.isfinite()], other[other.isfinite()], **tol)
    kernels.check_bounded_waits(DEV)


@pytest.mark.parametrize("blocks, bw", [(80, 72), (40, 136), (160, 8)])
def test_recurrent_gates_have_the_same_bits_in_tiles_of_every_height(blocks, bw):
    """Steps whose tiles are 16, 32, 64 and 128 rows high (`blocks` of channels enough for each), whole and part tiles."""
    from garlic_inference_b200.ops import kernels
    W = blocks * bw
    u = rnd(300, W, seed=1, scale=2.0)
    wa, wi = (rnd(blocks, bw, bw, seed=s, scale=bw ** -0.5, dtype=torch.bfloat16) for s in (2, 3))
    rest = wa, wi, rnd(W, seed=4), rnd(W, seed=5), rnd(W, seed=6), 8.0
    whole = kernels.rglru_gates(u, *rest)
    z = [torch.einsum("nbi,bio->nbo", u.double().view(300, blocks, bw), w.double()).reshape(300, W) + b.double()
         for w, b in ((wa, rest[2]), (wi, rest[3]))]
    log_a = -8.0 * torch.sigmoid(z[0]) * torch.nn.functional.softplus(rest[4].double())
    want = torch.exp(log_a), torch.sqrt(-torch.expm1(2 * log_a)) * torch.sigmoid(z[1]) * u.double()
    for got, w in zip(whole, want):
        assert (got.double() - w).norm() <= 1e-6 * w.norm()
    for at, n in ((0, 1), (3, 16), (17, 17), (20, 40), (100, 64), (64, 65), (0, 128), (170, 129)):
        for got, w in zip(kernels.rglru_gates(u[at:at + n].contiguous(), *rest), whole):
            assert torch.equal(got, w[at:at + n]), n


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


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("width", [40, 65, 130])
@pytest.mark.parametrize("first, row", [(0, 136), (8, 144), (4, 148), (2, 146), (1, 137), (3, 138), (0, 137)])
def test_recurrent_scan_over_columns_at_every_alignment(dtype, width, first, row):
    """y in columns whose rows start on 16, 8, 4 and 2 bytes, the same or another for every row: the bits of dense rows."""
    from garlic_inference_b200.ops import kernels
    lens = [70, 1, 6]
    n = sum(lens)
    a, b = torch.rand(n, width, generator=torch.Generator().manual_seed(1)).to(DEV), rnd(n, width, seed=2)
    wide = rnd(n, row, seed=3, dtype=dtype)
    y = wide[:, first:first + width]
    spans = torch.tensor([[i, sum(lens[:i]), m] for i, m in enumerate(lens)], dtype=torch.int32, device=DEV)
    slots, states = torch.zeros(n, dtype=torch.int32, device=DEV), [rnd(len(lens), width, seed=5) for _ in range(2)]
    padded = torch.zeros(n, -(-width // 8) * 8, dtype=dtype, device=DEV)
    padded[:, :width] = y                                                  # rows on 16 bytes
    want, got = (kernels.rglru_scan(a, b, v, None, s, spans, slots) for v, s in ((padded[:, :width], states[0]), (y, states[1])))
    assert torch.equal(got, want) and torch.equal(*states)
    one = torch.empty_like(wide)                                           # (a and b off 16 bytes as well)
    shifted = [torch.empty(n * width + 1, device=DEV)[1:].view(n, width).copy_(v) for v in (a, b)]
    out = kernels.rglru_scan(*shifted, y, None, rnd(len(lens), width, seed=5), spans, slots, out=one[:, first:first + width])
    assert torch.equal(out, want)


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


@pytest.mark.parametrize("N, K", [(1030, 1024), (2048, 516), (300, 3500)])
def test_float32_product_on_tensor_cores(N, K):
    """Weights of a million elements: rows on both sides of every tile height, inputs that are no whole slices, rows that lie
    apart and rows that do not start on 16 bytes: within the error of float32 sums, every row with the bits of its product alone."""
    from garlic_inference_b200.ops import kernels
    assert N * K >= kernels.SPLIT_MIN_ELEMENTS and K >= kernels.SPLIT_MIN_INPUTS
    w, full = rnd(N, K, seed=1), rnd(400, K + 5, seed=2)
    alone = {}
    for M in (1, 2, 15, 16, 17, 32, 33, 64, 65, 96, 97, 128, 129, 400):
        for a in (full[:M, :K].contiguous(), full[:M, :K]):
            out = torch.full((M, N + 3), 7.0, device=DEV)
            kernels.sgemm_nt_strided(a, w, out[:, :N])
            want = a.double() @ w.double().T
            tol = (K + 1) * 2.0 ** -24 * (a.double().abs() @ w.double().abs().T)       # a rounding an addition
            assert ((out[:, :N].double() - want).abs() <= tol).all() and bool((out[:, N:] == 7.0).all())
            for r in {0, M // 2, M - 1}:
                one = alone.setdefault(r, kernels.sgemm_nt(full[r:r + 1, :K].contiguous(), w)[0])
                assert torch.equal(out[r, :N], one), f"{M} rows, row {r}"
    kernels.check_bounded_waits(DEV)


@pytest.mark.parametrize("M, N, K", [(1, 130, 64), (16, 128, 68), (70, 257, 640), (200, 128, 1000)])
def test_every_form_of_the_float32_product_gives_the_same_bits(M, N, K):
    """All tile heights, with the inputs of a tile in one block and shared out; infinities, NaN and numbers that round up to an
    infinity come out as by multiply-adds."""
    from garlic_inference_b200.ops import kernels
    from garlic_inference_b200.ops.library import check, require_gpu
    l, flag = require_gpu(), kernels.tcgen05_error_flag(torch.device(DEV, 0))
    a, w = rnd(M, K, seed=3), rnd(N, K, seed=4)
    a[0, 5], a[M // 2, 9], a[M - 1, K - 1] = math.inf, math.nan, 3.4e38
    w[N - 1, 3], w[7, 11], w[9] = -math.inf, 3.4028234e38, 0.0
    want = torch.empty(M, N, device=DEV)
    check(l.gi_sgemm_nt(a.data_ptr(), w.data_ptr(), want.data_ptr(), M, N, K, K, N, 0), l)
    space = torch.empty(6 * M * (K + 8) + 4 * M * N * (K // 64 + 1) + 512, dtype=torch.uint8, device=DEV)
    first = None
    for tile in (16, 32, 64, 96, 128):
        for shares in (1, 3, 100):
            out = torch.full((M, N), 7.0, device=DEV)
            check(l.gi_sgemm_split_nt(a.data_ptr(), w.data_ptr(), out.data_ptr(), space.data_ptr(), space.numel(), M, N, K, K, N, tile, shares,
                                      flag.data_ptr(), 0), l)
            first = out if first is None else first
            assert torch.equal(out.view(torch.int32), first.view(torch.int32)), (tile, shares)
    odd = ~want.isfinite()
    assert torch.equal(first.isfinite(), want.isfinite()) and torch.equal(first[odd].isnan(), want[odd].isnan())
    assert torch.equal(first[odd & ~want.isnan()], want[odd & ~want.isnan()])
    with pytest.raises(Exception, match="work space"):
        check(l.gi_sgemm_split_nt(a.data_ptr(), w.data_ptr(), want.data_ptr(), space.data_ptr(), 16, M, N, K, K, N, 32, 1, flag.data_ptr(), 0), l)
    kernels.check_bounded_waits(DEV)


@pytest.mark.parametrize("a_scale, w_scale", [(1e-36, 1.0), (1e-40, 1e20), (1.0, 1e-36), (1e25, 1e-42), (1e-22, 1e-21), (1e13, 1e14), (1e30, 1e-3), (2e37, 1e-30)])
def test_float32_product_of_small_and_large_numbers(a_scale, w_scale):
    """Numbers from below the smallest normal one to near the largest, in every form: within the error of float32 sums, of results below the
    normal ones too."""
    from garlic_inference_b200.ops import kernels
    from garlic_inference_b200.ops.library import check, require_gpu
    l, flag, N, K = require_gpu(), kernels.tcgen05_error_flag(torch.device(DEV, 0)), 260, 640
    for M in (3, 70):
        a, w = rnd(M, K, seed=1, scale=a_scale), rnd(N, K, seed=2, scale=w_scale)
        want, tol = a.double() @ w.double().T, (K + 1) * 2.0 ** -24 * (a.double().abs() @ w.double().abs().T) + K * 2.0 ** -149
        space = torch.empty(6 * M * K + 4 * M * N * (K // 64) + 512, dtype=torch.uint8, device=DEV)
        for tile in (16, 32, 64, 96, 128):
            for shares in (1, 3):
                out = torch.full((M, N), 7.0, device=DEV)
                check(l.gi_sgemm_split_nt(a.data_ptr(), w.data_ptr(), out.data_ptr(), space.data_ptr(), space.numel(), M, N, K, K, N, tile, shares,
                                          flag.data_ptr(), 0), l)
                assert ((out.double() - want).abs() <= tol).all(), (M, tile, shares)


@pytest.mark.parametrize("space", [1 << 17, 1 << 20])
def test_float32_product_some_rows_at_a_time(space, monkeypatch):
    """Portions of 11 to 128 rows, as many as fit the work space or half and half again, rows that lie apart on both sides: every row's bits
    alone, the columns beside left alone, the launches counted."""
    from garlic_inference_b200.ops import kernels
    M, N, K = 300, 1030, 1024
    w, full = rnd(N, K, seed=1), rnd(M, K + 5, seed=2)
    alone = torch.cat([kernels.sgemm_nt(full[r:r + 1, :K].contiguous(), w) for r in range(M)])
    monkeypatch.setattr(kernels, "SPLIT_SPACE", space)
    l, out = kernels.require_gpu(), torch.full((M, N + 3), 7.0, device=DEV)
    before = kernels.counters.launches
    kernels.sgemm_nt_strided(full[:, :K], w, out[:, :N])
    want, r, parts = 0, 0, []
    while r < M:
        parts.append(min(M - r, 128))
        while parts[-1] > 16 and l.gi_sgemm_split_space(parts[-1], N, K) > space:
            parts[-1] = -(-parts[-1] // 2)
        want, r = want + l.gi_sgemm_split_launches(parts[-1], N, K), r + parts[-1]
    assert len(parts) > 2
    assert kernels.counters.launches - before == want
    assert torch.equal(out[:, :N], alone) and bool((out[:, N:] == 7.0).all())
    kernels.check_bounded_waits(DEV)


@pytest.mark.parametrize("M, N", [(5, 1000), (64, 512), (130, 260)])
def test_float32_product_of_long_rows(M, N):
    """Rings that go round many times in every form, with the sums kept and left in memory, W not in the L2 cache: the same bits time after
    time, within the error of float32 sums."""
    from garlic_inference_b200.ops import kernels
    from garlic_inference_b200.ops.library import check, require_gpu
    l, flag, K = require_gpu(), kernels.tcgen05_error_flag(torch.device(DEV, 0)), 17408
    a, w, other = rnd(M, K, seed=1), rnd(N, K, seed=2), torch.empty(256 << 20, dtype=torch.uint8, device=DEV)
    want = a.double() @ w.double().T
    tol = (K + 1) * 2.0 ** -24 * (a.double().abs() @ w.double().abs().T)               # a rounding an addition
    space = torch.empty(6 * M * K + 4 * M * N * (K // 64) + 512, dtype=torch.uint8, device=DEV)
    first = None
    for tile in (16, 32, 64, 96, 128):
        for shares in (1, 4, 9):
            for _ in range(4):
                other.zero_()
                out = torch.full((M, N), 7.0, device=DEV)
                check(l.gi_sgemm_split_nt(a.data_ptr(), w.data_ptr(), out.data_ptr(), space.data_ptr(), space.numel(), M, N, K, K, N, tile, shares,
                                          flag.data_ptr(), 0), l)
                first = out if first is None else first
                assert torch.equal(out, first), (tile, shares)
    assert ((first.double() - want).abs() <= tol).all()
    kernels.check_bounded_waits(DEV)


@pytest.mark.parametrize("M", [2097120, 2097121, 4194240])
@pytest.mark.parametrize("N", [3, 16])
def test_float32_product_of_millions_of_rows(M, N):
    """Around the rows that tiles of 32 take in one launch, and the most that are taken at all: the bits of a few rows."""
    from garlic_inference_b200.ops import KernelError, kernels
    K = 4
    a, w = torch.randn(M, K, generator=torch.Generator(device=DEV).manual_seed(1), device=DEV), rnd(N, K, seed=2)
    out = kernels.sgemm_nt(a, w)
    for at in (0, M // 2, M - 200):
        assert torch.equal(out[at:at + 200], kernels.sgemm_nt(a[at:at + 200].contiguous(), w))
    if M == 4194240:
        with pytest.raises(KernelError, match="rows"):
            kernels.sgemm_nt(torch.zeros(M + 1, 1, device=DEV), torch.zeros(1, 1, device=DEV))


# ---- tcgen05 prompt attention at sizes other than heads of 128 -------------------------------------------------------------
def _pools(lens, heads, d, page, seed, extra_pages=3):
    """(dense [len, heads, d] per sequence, pool, block table) with pages handed out in a mixed order."""
    need = [-(-n // page) for n in lens]
    order = torch.randperm(sum(need) + extra_pages, generator=torch.Generator().manual_seed(3)).tolist()
    pool = rnd(len(order), heads, page, d, seed=seed + 1, dtype=torch.bfloat16)
    table = torch.full((len(lens), max(need)), -1, dtype=torch.int32)
    dense = []
    for s, n in enumerate(lens):
        x = rnd(n, heads, d, seed=seed + 10 + s, dtype=torch.bfloat16)
        for lp in range(need[s]):
            table[s, lp] = order.pop()
            part = x[lp * page:(lp + 1) * page]
            pool[int(table[s, lp]), :, :len(part)] = part.transpose(0, 1)
        dense.append(x)
    return dense, pool, table.to(DEV)


def _runs128(lens, new):
    from garlic_inference_b200.parts import StepShape
    from garlic_inference_b200.parts.attention import query_runs
    starts = [sum(new[:i]) for i in range(len(new))]
    shape = StepShape(list(range(len(lens))), starts, new, [n - m for n, m in zip(lens, new)], False)
    return torch.from_numpy(query_runs(shape, 128)).to(DEV), starts


def _attend64(q, k, v, pos0, scale, window=0, chunk=0, keep=0, sink=None, bias=None):
    """q [m, d] of one head at positions pos0 .., k [n, d], v [n, dv] in 64 bits."""
    i = pos0 + torch.arange(q.shape[0], device=DEV)[:, None]
    j = torch.arange(k.shape[0], device=DEV)[None]
    seen = (j <= i) & ((i - j < window) | (j < keep) if window else True) & ((i // chunk == j // chunk) if chunk else True)
    s = q.double() @ k.double().T * scale
    if bias is not None:
        s = s + bias.double()[(i - j).clamp(0, len(bias) - 1)]
    s = s.masked_fill(~seen, -math.inf)
    top = s.max(-1, keepdim=True).values if sink is None else torch.maximum(s.max(-1, keepdim=True).values, sink.double())
    e = torch.exp(s - top)
    return e @ v.double() / (e.sum(-1, keepdim=True) + (0.0 if sink is None else torch.exp(sink.double() - top)))


# the probabilities' rounding to 8 bits (2^-8 of a weighted mean of values of size 1, up to 4 here), their exponent's and the
# result's own: one part in 100 of the largest value
ATT_TOL = dict(rtol=2e-2, atol=2e-2)


@pytest.mark.parametrize("d, dv, maps, n_dist, page", [(64, 64, 1, 0, 64), (64, 128, 2, 0, 64), (64, 128, 1, 0, 128), (128, 64, 1, 0, 64),
                                                       (128, 64, 1, 90, 64), (64, 64, 1, 700, 128), (128, 128, 1, 1, 64), (64, 64, 2, 0, 64)])
@pytest.mark.parametrize("mask", [{}, {"window": 70}, {"window": 33, "keep_first": 70}, {"chunk": 100}])
def test_prompt_attention_on_tensor_memory_at_other_sizes(d, dv, maps, n_dist, page, mask):
    """Tiles that are and are not whole, portions behind cached tokens, every mask, several maps per head, tables of biases
    shorter and longer than the sequences, sinks and gates where they are taken."""
    from garlic_inference_b200.ops import kernels
    H, G = 6, 2
    lens, new = [1, 37, 300, 64, 65, 513], [1, 37, 250, 64, 3, 513]
    assert kernels.tcgen05_attention_takes(torch.bfloat16, d, page, dv, n_dist=n_dist)
    ks, k_pool, table = _pools(lens, G * maps, d, page, 20)
    vs, v_pool, _ = _pools(lens, G, dv, page, 60)
    runs, starts = _runs128(lens, new)
    n, scale = sum(new) + 2, d ** -0.5                                     # two rows in no tile
    q = rnd(n, H * maps, d, seed=5, dtype=torch.bfloat16)
    bias = rnd(n_dist, H, seed=6) if n_dist else None
    for sinks, gate in [(None, None)] + ([(rnd(H, seed=7), None)] if maps == 1 else []) + \
            ([(None, rnd(n, H, seed=8, dtype=torch.bfloat16)), (None, rnd(n, H * dv, seed=9, dtype=torch.bfloat16))]
             if maps == 1 and not n_dist and (d, dv) != (64, 128) else []):
        kw = dict(sinks=sinks, gate=gate, maps=maps, dist_bias=bias, chunk=mask.get("chunk", 0), keep_first=mask.get("keep_first", 0))
        got = kernels.attention_prefill_tcgen05(q, k_pool, v_pool, table, runs, scale, mask.get("window", 0), **kw).view(n, H * maps, dv)
        assert float(got[-2:].abs().max()) == 0.0
        wide = torch.full((n, H * maps * dv + 8), 3.0, dtype=torch.bfloat16, device=DEV)      # into columns of a wider matrix
        kernels.attention_prefill_tcgen05(q, k_pool, v_pool, table, runs, scale, mask.get("window", 0), out=wide[:, 8:], **kw)
        assert torch.equal(wide[:-2, 8:].reshape(-1), got[:-2].reshape(-1)) and bool((wide[:, :8] == 3.0).all()) and bool((wide[-2:] == 3.0).all())
        for s, (at, m) in enumerate(zip(starts, new)):
            for hh in range(H * maps):
                h, g = hh // maps, hh // maps // (H // G)
                want = _attend64(q[at:at + m, hh], ks[s][:, g * maps + hh % maps], vs[s][:, g], lens[s] - m, scale,
                                 mask.get("window", 0), mask.get("chunk", 0), mask.get("keep_first", 0),
                                 None if sinks is None else sinks[h], None if bias is None else bias[:, h])
                if gate is not None:
                    want = want * torch.sigmoid((gate if gate.shape[1] == H * dv else gate.repeat_interleave(dv, 1))[at:at + m, h * dv:(h + 1) * dv].double())
                torch.testing.assert_close(got[at:at + m, hh].double(), want, **ATT_TOL)
    kernels.check_bounded_waits(torch.device("cuda", 0))


@pytest.mark.parametrize("d, dv, maps, n_dist, rot", [(64, 64, 1, 0, False), (64, 128, 2, 0, False), (128, 64, 1, 0, False),
                                                      (128, 128, 1, 0, False), (128, 128, 1, 0, True), (64, 64, 1, 90, False)])
@pytest.mark.parametrize("window", [0, 50])
def test_prompt_attention_beside_what_a_page_held_before(d, dv, maps, n_dist, rot, window):
    """Infinities and NaN behind a sequence's last token (left in its page by the page's owner before) reach no result."""
    from garlic_inference_b200.ops import kernels
    H, G, page = (3, 3, 128) if rot else (4, 2, 128)
    lens, new = ([300], [70]) if rot else ([1, 37, 300, 64, 65, 513, 128], [1, 37, 70, 64, 3, 513, 100])
    if rot:
        page = 320
    ks, k_pool, table = _pools(lens, G * maps, d, page, 20, extra_pages=0)
    vs, v_pool, _ = _pools(lens, G, dv, page, 60, extra_pages=0)
    shared = rnd(page, 64, seed=4, dtype=torch.bfloat16) if rot else None
    runs, starts = _runs128(lens, new)
    q = rnd(sum(new), H * maps, d + 64 * rot, seed=5, dtype=torch.bfloat16)
    bias = rnd(n_dist, H, seed=6) if n_dist else None
    run = lambda: kernels.attention_prefill_tcgen05(q, k_pool, v_pool, table, runs, d ** -0.5, window, maps=maps, dist_bias=bias,
                                                    rows_covered=True, **({"rot": (shared, 0)} if rot else {}))
    for pool in (k_pool, v_pool):                                          # zeros behind the ends, then anything
        for s, n in enumerate(lens):
            if n % page:
                pool[int(table[s, n // page]), :, n % page:] = 0.0
    want = run()
    for pool, bad in ((k_pool, (math.nan, math.inf)), (v_pool, (math.inf, math.nan))):
        for s, n in enumerate(lens):
            if n % page:
                pool[int(table[s, n // page]), :, n % page:, ::2], pool[int(table[s, n // page]), :, n % page:, 1::2] = bad
    if rot:
        shared[lens[0]:] = math.nan
    assert torch.isfinite(want).all() and torch.equal(run(), want)
    kernels.check_bounded_waits(torch.device("cuda", 0))


@pytest.mark.parametrize("n_dist", [40, 500])
def test_distance_biases_where_a_block_walks_many_items(n_dist):
    """More than six items of different heads to every persistent block, each with a table of its own in the same place."""
    from garlic_inference_b200.ops import kernels
    H, G, d, dv, page = 40, 8, 128, 64, 64
    new = [1 + (37 * i) % 131 for i in range(44)]
    lens = [m + (29 * i) % 90 for i, m in enumerate(new)]
    ks, k_pool, table = _pools(lens, G, d, page, 20)
    vs, v_pool, _ = _pools(lens, G, dv, page, 90)
    runs, starts = _runs128(lens, new)
    assert runs.shape[0] * H > 6 * 2 * 148
    q, bias = rnd(sum(new), H, d, seed=5, dtype=torch.bfloat16), rnd(n_dist, H, seed=6)
    got = kernels.attention_prefill_tcgen05(q, k_pool, v_pool, table, runs, d ** -0.5, 0, dist_bias=bias).view(-1, H, dv)
    for s, (at, m) in enumerate(zip(starts, new)):
        for h in range(H):
            want = _attend64(q[at:at + m, h], ks[s][:, h * G // H], vs[s][:, h * G // H], lens[s] - m, d ** -0.5, bias=bias[:, h])
            torch.testing.assert_close(got[at:at + m, h].double(), want, **ATT_TOL)
    kernels.check_bounded_waits(torch.device("cuda", 0))


@pytest.mark.parametrize("past, m", [(0, 1), (0, 129), (63, 70), (300, 40)])
@pytest.mark.parametrize("window", [0, 90])
def test_prompt_attention_with_a_key_part_that_all_heads_share(past, m, window):
    """Keys of 128 and a shared part of 64 in columns of rows of their own, with a sink and a gate per head."""
    from garlic_inference_b200.ops import kernels
    H, T, scale = 3, past + m, 192 ** -0.5
    pad = -(-T // 64) * 64
    k, v, rows = (rnd(*shape, seed=i, dtype=torch.bfloat16) for i, shape in enumerate([(1, H, pad, 128), (1, H, pad, 128), (pad, 88)]))
    q, gate, sinks = rnd(m, H, 192, seed=4, dtype=torch.bfloat16), rnd(m, H, seed=5, dtype=torch.bfloat16), rnd(H, seed=6)
    table = torch.zeros((1, 1), dtype=torch.int32, device=DEV)
    runs, _ = _runs128([T], [m])
    got = kernels.attention_prefill_tcgen05(q, k, v, table, runs, scale, window, rot=(rows, 16), gate=gate, sinks=sinks).view(m, H, 128)
    for h in range(H):
        want = _attend64(q[:, h], torch.cat([k[0, h, :T], rows[:T, 16:80]], -1), v[0, h, :T], past, scale, window, sink=sinks[h])
        torch.testing.assert_close(got[:, h].double(), want * torch.sigmoid(gate[:, h:h + 1].double()), **ATT_TOL)
    kernels.check_bounded_waits(torch.device("cuda", 0))


# ---- latent attention: portions whose keys and values are expanded beside a rotated part -----------------------------------
@pytest.mark.parametrize("layout, q_rank, gate, sink, pad", [("half", 24, True, False, 0), ("interleaved", 0, False, True, 8),
                                                             ("half", 24, True, True, 3)])
@pytest.mark.parametrize("lens, past", [([130], [0]), ([200, 3, 64, 129], [70, 10, 0, 300]), ([127, 128], [0, 1])])
def test_latent_portions_with_a_rotated_part(layout, q_rank, gate, sink, pad, lens, past):
    """Portions on both sides of the length from which keys and values are expanded, alone and in one step, whole and behind
    cached tokens; into columns of a wider matrix that do and do not start on 16 bytes (`pad`); against 64 bits."""
    from garlic_inference_b200.cache import PagedCache
    from garlic_inference_b200.parts import RotaryPositions, Runtime, StepContext
    from garlic_inference_b200.parts.latent_attention import LatentAttention
    H, hid, r, d, dr, dv = 3, 64, 40, 128, 64, 128
    params = dict(hidden_size=hid, n_heads=H, plain_dim=d, rot_dim=dr, value_dim=dv, kv_rank=r, q_rank=q_rank,
                  softmax_scale=0.07, eps=1e-6, head_gate=gate, sink=sink, own_kv=True)
    w = {n: rnd(*t.shape, seed=i, scale=t.shape[-1] ** -0.5 if len(t.shape) > 1 else 1.0, dtype=torch.bfloat16)
         for i, (n, t) in enumerate(sorted(LatentAttention.wanted(params).items()))}

    class Load:
        def dtype(self, *names):
            return torch.bfloat16

        def __call__(self, n, out=None):
            return w[n] if out is None else out.copy_(w[n])

    rt = Runtime(torch.bfloat16, torch.device("cuda", 0))
    part = LatentAttention(params, Load(), rt)
    rot = RotaryPositions(dict(head_dim=dr, rotary_dim=dr, theta=1e4, max_positions=1024, layout=layout, tables=False), None, rt)
    cache = PagedCache([part.cache_requirement()], max_tokens=2048, max_positions=1024, dtype=torch.bfloat16, device="cuda")
    xs = [rnd(p + m, hid, seed=90 + i, dtype=torch.bfloat16) for i, (m, p) in enumerate(zip(lens, past))]
    slots = [cache.alloc_slot() for _ in lens]

    def run(ns, befores, **kw):
        which = [i for i, m in enumerate(ns) if m]
        s, ns, befores = [slots[i] for i in which], [ns[i] for i in which], [befores[i] for i in which]
        cache.prepare(s, ns)
        cat = lambda f: torch.cat([torch.as_tensor(f(i), dtype=torch.int32) for i in range(len(s))]).to(DEV)
        n = sum(ns)
        ctx = StepContext(n, torch.zeros(n, dtype=torch.int32, device=DEV), cat(lambda i: torch.arange(befores[i], befores[i] + ns[i])),
                          cat(lambda i: torch.full((ns[i],), s[i])), s, [sum(ns[:i]) for i in range(len(s))], ns, befores, False,
                          1024, status=cache.status)
        x = torch.cat([xs[i][befores[j]:befores[j] + ns[j]] for j, i in enumerate(which)])
        y = part.pre_output(x, ctx, cache.view(0), rot, True, **kw)
        cache.commit(s, ns)
        return y

    if any(past):
        run(past, [0] * len(past))
    n = sum(lens)
    wide = torch.zeros((n, H * dv + 16), dtype=torch.bfloat16, device=DEV)
    got = run(lens, past) if pad == 0 else run(lens, past, out=wide[:, pad:pad + H * dv])
    f = 1e4 ** (-2.0 * torch.arange(dr // 2, dtype=torch.float64, device=DEV) / dr)

    def turn(x):
        a = torch.arange(x.shape[0], dtype=torch.float64, device=DEV)[:, None, None] * f
        u, v = (x[..., :dr // 2], x[..., dr // 2:]) if layout == "half" else (x[..., ::2], x[..., 1::2])
        u, v = u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin()
        return torch.cat([u, v], -1) if layout == "half" else torch.stack([u, v], -1).flatten(-2)

    W = {k: v.double() for k, v in w.items()}
    rms = lambda x, g: x / torch.sqrt((x * x).mean(-1, keepdim=True) + 1e-6) * g
    at = 0
    for x, m, p in zip(xs, lens, past):
        x, T = x.double(), len(x)
        q = ((rms(x @ W["dq"].T, W["dq.norm"]) @ W["uq"].T) if q_rank else x @ W["q"].T).view(T, H, d + dr)
        c = x @ W["dkv"].T
        c, kr = rms(c[:, :r], W["dkv.norm"]), turn(c[:, None, r:])[:, 0]
        k, v = (c @ W["uk"].T).view(T, H, d), (c @ W["uv"].T).view(T, H, dv)
        q = torch.cat([q[..., :d], turn(q[..., d:])], -1)
        for h in range(H):
            want = _attend64(q[p:, h], torch.cat([k[:, h], kr], -1), v[:, h], p, 0.07, sink=W["sink"][h] if sink else None)
            if gate:
                want = want * torch.sigmoid(x[p:] @ W["g"][h])[:, None]
            # beside the attention's own roundings those of q, k, v and the latents (2^-9 each of values of size 1 to 4)
            torch.testing.assert_close(got[at:at + m].view(m, H, dv)[:, h].double() if pad == 0 else
                                       got[at:at + m, h * dv:(h + 1) * dv].double(), want, rtol=4e-2, atol=4e-2)
        at += m
    cache.check_status()


# ---- row-wise kernels that move words of four ----------------------------------------------------------------------------------
@pytest.mark.parametrize("layout, q_rank, gate, sink, pad", [("half", 24, True, False, 0), ("interleaved", 0, False, True, 8)])
def test_latent_portions_expanded_beside_others_that_are_not(layout, q_rank, gate, sink, pad, monkeypatch):
    """The step of four portions above with every portion that may be expanded so, whatever it gains: two are, two are not.  And
    the choice itself: beside other portions only those of many scores, alone all of them."""
    from types import SimpleNamespace
    from garlic_inference_b200.parts import StepShape
    from garlic_inference_b200.parts import latent_attention
    from garlic_inference_b200.parts.latent_attention import LatentAttention
    monkeypatch.setattr(latent_attention, "MIXED_MIN_SCORES", 0)
    test_latent_portions_with_a_rotated_part(layout, q_rank, gate, sink, pad, [200, 3, 64, 129], [70, 10, 0, 300])
    monkeypatch.undo()
    part = SimpleNamespace(dr=64, d=128, dv=128, rank=512, H=32, window=0, rt=SimpleNamespace(dtype=torch.bfloat16),
                           w_uv=torch.zeros(1, dtype=torch.bfloat16), w_uk_t=torch.zeros(1, dtype=torch.bfloat16))
    for name in ("_expands", "_first_page", "_first_seen", "_run_rows", "_runs_name"):
        setattr(part, name, getattr(LatentAttention, name).__get__(part))
    chosen = lambda lens, past: [w[0] for w in LatentAttention._portions(part, StepShape([], [], lens, past, False), 64)]
    assert chosen([200], [70]) == [0] and chosen([200, 40], [70, 0]) == [0, 1]
    assert chosen([200, 3], [70, 10]) == [] and chosen([3, 200, 512], [10, 70, 512]) == [2]      # 32 x 512 x 1,024 scores: the line


@pytest.mark.parametrize("bytes_, pad", [(1, 0), (2 * 2 * 512 * 256, 8)])
def test_latent_portions_expanded_some_heads_at_a_time(bytes_, pad, monkeypatch):
    """One head at a time and, with 512 keys, two and then one of three, with gates and sinks; whole rows and columns."""
    from garlic_inference_b200.parts import latent_attention
    monkeypatch.setattr(latent_attention, "EXPAND_RUN_BYTES", bytes_)
    test_latent_portions_with_a_rotated_part("half", 24, True, True, pad, [130, 200], [0, 300])


def test_latent_portions_need_no_more_memory_than_their_scores_did():
    """A portion behind 60,000 cached tokens, 32 heads: 1 GB of keys and values in all, at most 256 MB of them at a time."""
    from garlic_inference_b200.parts import Runtime, StepContext, latent_attention
    from garlic_inference_b200.parts.latent_attention import LatentAttention
    H, hid, r, past, new, page = 32, 64, 64, 60000, 128, 64
    params = dict(hidden_size=hid, n_heads=H, plain_dim=128, rot_dim=64, value_dim=128, kv_rank=r, q_rank=0, softmax_scale=0.07,
                  eps=1e-6, head_gate=False, own_kv=True)

    class Load:
        def dtype(self, *names):
            return torch.bfloat16

        def __call__(self, n, out=None):
            t = rnd(*LatentAttention.wanted(params)[n].shape, seed=len(n), scale=0.1, dtype=torch.bfloat16)
            return t if out is None else out.copy_(t)

    part = LatentAttention(params, Load(), Runtime(torch.bfloat16, torch.device("cuda", 0)))
    pages = -(-(past + new) // page)
    from types import SimpleNamespace
    kv = SimpleNamespace(page_size=page, k_pool=rnd(pages, 1, page, part.row, seed=1, dtype=torch.bfloat16),
                         block_table=torch.arange(pages, dtype=torch.int32, device=DEV).view(1, -1))
    ctx = StepContext(new, *(torch.zeros(new, dtype=torch.int32, device=DEV) for _ in range(3)), [0], [0], [new], [past], False, past + new)
    which = part._portions(ctx, page)
    assert len(which) == 1
    q, out = rnd(new, H, 192, seed=2, dtype=torch.bfloat16), torch.zeros(new, H * 128, dtype=torch.bfloat16, device=DEV)
    part._attend_expanded(q, kv, ctx, which, None, out)                     # (the library's workspace is made)
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    part._attend_expanded(q, kv, ctx, which, None, out)
    gathered = pages * page * part.row * 2
    assert torch.cuda.max_memory_allocated() - before <= (256 << 20) + 2 * gathered + (4 << 20)


@pytest.mark.parametrize("hidden", [4, 100, 1024, 4100, 9000, 6])
@pytest.mark.parametrize("n", [1, 300])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_embedding_rows(hidden, n, dtype):
    from garlic_inference_b200.ops import kernels
    table = rnd(50, hidden, seed=1, dtype=dtype)
    ids = torch.randint(0, 50, (n,), generator=torch.Generator().manual_seed(2)).to(torch.int32).to(DEV)
    ids[0] = 50                                                            # outside the vocabulary: zeros
    want = table.float()[ids.clamp(max=49).long()] * 0.5
    want[0] = 0.0
    assert torch.equal(kernels.embedding(ids, table, scale=0.5), want)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("groups, gs, pad", [(3, 4, 0), (5, 132, 4), (2, 512, 0), (1, 516, 0), (3, 10, 2), (4, 128, 1)])
@pytest.mark.parametrize("n", [1, 37])
def test_norms_of_groups_and_heads_with_gates(dtype, groups, gs, pad, n):
    """The read-out's norm per group and the attention's finish per head, sizes on both sides of a warp's words and rows that
    do and do not start on them."""
    from garlic_inference_b200.ops import kernels
    tol = dict(rtol=2e-5, atol=1e-5) if dtype == torch.float32 else dict(rtol=2.0 ** -7, atol=1e-3)      # one rounding of the result
    W = groups * gs
    o, g = rnd(n, W, seed=1), rnd(n, W + pad, seed=2, dtype=dtype)[:, :W]
    w = rnd(gs, seed=3, dtype=dtype)
    out = torch.full((n, W + pad), 5.0, dtype=dtype, device=DEV)
    kernels.gated_group_rmsnorm(o, g, w, 1e-5, groups=groups, gate_kind="silu", mul=0.7, out=out[:, pad:])
    x = o.double().view(n, groups, gs)
    x = (x / torch.sqrt((x * x).mean(-1, keepdim=True) + 1e-5) * w.double()).view(n, W) * torch.nn.functional.silu(g.double()) * 0.7
    torch.testing.assert_close(out[:, pad:].double(), x, **tol)
    assert bool((out[:, :pad] == 5.0).all())
    lam = torch.tensor([0.3], device=DEV)
    for maps, gate in ((2, rnd(n, groups + 1, seed=4, dtype=dtype)[:, 1:]), (1, g), (2, None)):
        att = rnd(n, groups * maps * gs, seed=5, dtype=dtype)
        got = kernels.attn_finish(att, groups, maps, lam if maps == 2 else None, 1e-5, 0.4, gate, dtype, out=out[:, pad:])
        a = att.double().view(n, groups, maps, gs)
        a = a[:, :, 0] - lam.double() * a[:, :, 1] if maps == 2 else a[:, :, 0]
        a = a / torch.sqrt((a * a).mean(-1, keepdim=True) + 1e-5) * 0.4
        if gate is not None:
            a = a * torch.sigmoid(gate.double().view(n, groups, -1))
        torch.testing.assert_close(got.double(), a.view(n, W), **tol)


# ---- delta rule over prompts ------------------------------------------------------------------------------------------------------
@pytest.mark.parametrize("channel", [False, True])
@pytest.mark.parametrize("d, dv, H, Hk", [(128, 128, 16, 8), (64, 128, 20, 20), (64, 16, 3, 3), (128, 48, 2, 1)])
@pytest.mark.parametrize("lens", [[8], [1, 7, 9, 64], [33, 100, 2, 16]])
def test_delta_rule_by_two_kernels_has_the_bits_of_one(channel, d, dv, H, Hk, lens, monkeypatch):
    """Sequences of whole and part groups of tokens, shorter than the ring, a padding portion; against the kernel that decode
    steps run (bits) and against 64 bits."""
    from garlic_inference_b200.ops import kernels
    n, n_dec = sum(lens) + 2, H * d if channel else H
    qkv, ab, al = rnd(n, 2 * Hk * d + H * dv, seed=1), rnd(n, 2 * H, seed=2), rnd(n, n_dec, seed=3)
    A_log, dt = rnd(H, seed=4, scale=0.3), rnd(n_dec, seed=5)
    starts = [sum(lens[:i]) for i in range(len(lens))]
    spans = torch.tensor([[i, s, m] for i, (s, m) in enumerate(zip(starts, lens))] + [[-1, n - 2, 2]], dtype=torch.int32, device=DEV)
    slots = torch.zeros(n, dtype=torch.int32, device=DEV)
    first = rnd(len(lens) + 1, H * dv * d + 8, seed=6, scale=0.1)

    def run(pair):
        monkeypatch.setattr(kernels, "DELTA_PAIR_TOKENS", 0 if pair else 1 << 30)
        state = first.clone()
        out = kernels.delta_scan(qkv, (0, Hk * d, 2 * Hk * d), ab, (H, 0), A_log, dt, state, spans, slots, H, Hk, d, dv, 1e-6,
                                 channel_decay=channel, decay_logits=al)
        return out, state

    (got, state), (one, state1) = run(True), run(False)
    assert torch.equal(got, one) and torch.equal(state, state1)
    assert float(got[n - 2:].abs().max()) == 0.0
    q, k, v = (qkv[:, a:b].double() for a, b in ((0, Hk * d), (Hk * d, 2 * Hk * d), (2 * Hk * d, 2 * Hk * d + H * dv)))
    unit = lambda x: (x.view(n, Hk, d) / torch.sqrt((x.view(n, Hk, d) ** 2).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // Hk, 1)
    q, k, v, beta = unit(q) * d ** -0.5, unit(k), v.view(n, H, dv), torch.sigmoid(ab[:, H:].double())
    g = torch.exp(-torch.exp(A_log.double())[:, None] * torch.nn.functional.softplus(al.double() + dt.double()).view(n, H, -1))
    for i, (s, m) in enumerate(zip(starts, lens)):
        S = first[i, :H * dv * d].double().view(H, dv, d)
        for t in range(s, s + m):
            S = S * g[t][:, None, :]
            u = beta[t][:, None] * (v[t] - (S @ k[t][:, :, None])[..., 0])
            S = S + u[:, :, None] * k[t][:, None, :]
            torch.testing.assert_close(got[t].view(H, dv).double(), (S @ q[t][:, :, None])[..., 0], rtol=1e-4, atol=1e-5)


@pytest.mark.parametrize("channel", [False, True])
@pytest.mark.parametrize("lens", [[200], [33, 100, 2, 16], [64, 64, 9]])
def test_delta_rule_by_two_kernels_some_rows_at_a_time(channel, lens, monkeypatch):
    """The same bits where the step's rows pass what is kept of them at a time (64 here): sequences cut in one and in two places,
    at a cut's edge, and wholly behind it."""
    from garlic_inference_b200.ops import kernels
    monkeypatch.setattr(kernels, "DELTA_SCRATCH_BYTES", 1)
    test_delta_rule_by_two_kernels_has_the_bits_of_one(channel, 64, 16, 3, 3, lens, monkeypatch)
    test_delta_rule_by_two_kernels_has_the_bits_of_one(channel, 128, 48, 2, 1, lens, monkeypatch)


@pytest.mark.parametrize("channel", [False, True])
@pytest.mark.parametrize("d, dv, H, Hk", [(128, 128, 4, 2), (64, 16, 3, 3), (128, 144, 2, 1)])
@pytest.mark.parametrize("lens, at_a_time", [([1, 15, 16, 17, 33], None), ([100], None), ([70, 3, 64], 40)])
def test_delta_rule_in_chunks(channel, d, dv, H, Hk, lens, at_a_time, monkeypatch):
    """Part chunks, a padding portion, decays of zero and of one, a step cut into rows that are taken at a time: against 64 bits, as
    close as token by token."""
    from garlic_inference_b200.ops import kernels
    from garlic_inference_b200.ops.library import require_gpu
    n, n_dec = sum(lens) + 2, H * d if channel else H
    qkv, ab, al = rnd(n, 2 * Hk * d + H * dv, seed=1), rnd(n, 2 * H, seed=2), rnd(n, n_dec, seed=3, scale=2.0)
    al[1], al[2, 0] = 1e4, -1e4                                  # a decay of zero, one of one
    A_log, dt = rnd(H, seed=4, scale=0.3), rnd(n_dec, seed=5) - 2.0
    starts = [sum(lens[:i]) for i in range(len(lens))]
    spans = torch.tensor([[i, s, m] for i, (s, m) in enumerate(zip(starts, lens))] + [[-1, n - 2, 2]], dtype=torch.int32, device=DEV)
    slots = torch.zeros(n, dtype=torch.int32, device=DEV)
    first = rnd(len(lens) + 1, H * dv * d + 8, seed=6, scale=0.1)
    if at_a_time:
        monkeypatch.setattr(kernels, "DELTA_SCRATCH_BYTES", require_gpu().gi_delta_chunk_bytes(H, d, dv) * (len(lens) + 1 + at_a_time // 16))
        monkeypatch.setattr(kernels, "DELTA_CHUNK_ROWS", 16)

    def run(chunks):
        monkeypatch.setattr(kernels, "DELTA_CHUNK_TOKENS", 0)
        state, launched = first.clone(), kernels.counters.launches
        out = kernels.delta_scan(qkv, (0, Hk * d, 2 * Hk * d), ab, (H, 0), A_log, dt, state, spans, slots, H, Hk, d, dv, 1e-6,
                                 channel_decay=channel, decay_logits=al, chunks=chunks)
        return out, state, kernels.counters.launches - launched

    got, state, launched = run(True)
    one, state1, _ = run(False)
    assert launched == 2 * (-(-n // (at_a_time // 16 * 16)) if at_a_time else 1)
    assert not torch.equal(got, one) and float(got[n - 2:].abs().max()) == 0.0 and torch.equal(state[:, H * dv * d:], first[:, H * dv * d:])
    q, k, v = (qkv[:, a:b].double() for a, b in ((0, Hk * d), (Hk * d, 2 * Hk * d), (2 * Hk * d, 2 * Hk * d + H * dv)))
    unit = lambda x: (x.view(n, Hk, d) / torch.sqrt((x.view(n, Hk, d) ** 2).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // Hk, 1)
    q, k, v, beta = unit(q) * d ** -0.5, unit(k), v.view(n, H, dv), torch.sigmoid(ab[:, H:].double())
    g = torch.exp(-torch.exp(A_log.double())[:, None] * torch.nn.functional.softplus(al.double() + dt.double()).view(n, H, -1))
    want, last = torch.zeros(n, H, dv, dtype=torch.float64, device=DEV), first.double()
    for i, (s, m) in enumerate(zip(starts, lens)):
        S = first[i, :H * dv * d].double().view(H, dv, d)
        for t in range(s, s + m):
            S = S * g[t][:, None, :]
            u = beta[t][:, None] * (v[t] - (S @ k[t][:, :, None])[..., 0])
            S = S + u[:, :, None] * k[t][:, None, :]
            want[t] = (S @ q[t][:, :, None])[..., 0]
        last[i, :H * dv * d] = S.reshape(-1)
    far = lambda x, y: float((x.double() - y).norm() / y.norm())
    # some eight roundings to 2^-24 of a number between unit vectors and a result; token by token they are as many
    for x, x1, y in ((got, one, want.view(n, -1)), (state, state1, last)):
        assert far(x, y) < 8 * 2.0 ** -24 and far(x, y) < 2.0 * far(x1, y) + 2.0 ** -24
    kernels.check_bounded_waits(DEV)


def _delta_case(n, H, d, dv, channel, seed=1, center=-2.0, spread=2.0):
    """One sequence: (rows, logits of beta, logits of the decay, A_log, dt_bias, first state), one key head a head."""
    n_dec = H * d if channel else H
    return (rnd(n, 2 * H * d + H * dv, seed=seed), rnd(n, H, seed=seed + 1), rnd(n, n_dec, seed=seed + 2, scale=spread),
            rnd(H, seed=seed + 3, scale=0.3), rnd(n_dec, seed=seed + 4) + center, rnd(1, H * dv * d, seed=seed + 5, scale=0.1))


def _delta_run(case, H, d, dv, channel, chunks, eps=1e-6):
    from garlic_inference_b200.ops import kernels
    qkv, beta, al, A_log, dt, first = case
    n, state = qkv.shape[0], first.clone()
    spans = torch.tensor([[0, 0, n]], dtype=torch.int32, device=DEV)
    out = kernels.delta_scan(qkv, (0, H * d, 2 * H * d), beta, (0, 0), A_log, dt, state, spans, torch.zeros(n, dtype=torch.int32, device=DEV),
                             H, H, d, dv, eps, channel_decay=channel, decay_logits=al, chunks=chunks)
    kernels.check_bounded_waits(DEV)
    return out.view(n, H, dv), state.view(H, dv, d)


@pytest.mark.parametrize("channel", [False, True])
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("n", [17, 31, 32])
def test_delta_rule_in_chunks_without_an_addend_under_the_roots(channel, d, n, monkeypatch):
    """unit_eps of zero: the tokens that fill a part chunk up are zeros all the same."""
    from garlic_inference_b200.ops import kernels
    monkeypatch.setattr(kernels, "DELTA_CHUNK_TOKENS", 0)
    case = _delta_case(n, 2, d, 32, channel)
    for got, one in zip(_delta_run(case, 2, d, 32, channel, True, 0.0), _delta_run(case, 2, d, 32, channel, False, 0.0)):
        # each within eight roundings to 2^-24 of the result (test_delta_rule_in_chunks)
        assert bool(got.isfinite().all()) and float((got - one).norm() / one.norm()) < 16 * 2.0 ** -24


@pytest.mark.parametrize("channel", [False, True])
@pytest.mark.parametrize("d, n", [(64, 40), (128, 47)])
@pytest.mark.parametrize("what, at", [("v", 20), ("v", 16), ("v", 31), ("k", 25), ("q", 30), ("beta", 9), ("decay", 37)])
@pytest.mark.parametrize("value", [math.inf, -math.inf, math.nan])
def test_delta_rule_in_chunks_keeps_later_tokens_out_of_earlier_outputs(channel, d, n, what, at, value, monkeypatch):
    """One number beyond the finite inside a chunk: the outputs that are finite token by token are so in chunks, with the same values, and
    no others."""
    from garlic_inference_b200.ops import kernels
    monkeypatch.setattr(kernels, "DELTA_CHUNK_TOKENS", 0)
    H, dv = 2, 32
    case = _delta_case(n, H, d, dv, channel)
    qkv, beta, al = case[:3]
    {"q": qkv[:, 5:], "k": qkv[:, H * d + 5:], "v": qkv[:, 2 * H * d + 5:], "beta": beta, "decay": al}[what][at, 0] = value
    (got, state), (one, state1) = _delta_run(case, H, d, dv, channel, True), _delta_run(case, H, d, dv, channel, False)
    assert bool(one[:at].isfinite().all()) and bool(one[:, 1].isfinite().all())
    for x, y in ((got, one), (state, state1)):
        fine = y.isfinite()
        assert torch.equal(x.isfinite(), fine)
        # each within eight roundings to 2^-24 of the result (test_delta_rule_in_chunks)
        assert float((x - y)[fine].norm() / y[fine].norm()) < 16 * 2.0 ** -24


@pytest.mark.parametrize("channel", [False, True])
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("center, share", [(-9.0, 0.25), (-4.0, 0.8), (-2.0, 1.0), (0.0, 1.1), (3.0, 1.1)])
def test_delta_rule_in_chunks_is_as_close_to_64_bits_as_token_by_token(channel, d, center, share, monkeypatch):
    """From decays near 1 (long memories: token by token every rounded decay adds its error, in chunks one rounded product of 16) to states
    that are forgotten within a token, where both round a result a few times (a tenth for what is not the same number of times)."""
    from garlic_inference_b200.ops import kernels
    monkeypatch.setattr(kernels, "DELTA_CHUNK_TOKENS", 0)
    n, H, dv = 600, 4, 64
    case = _delta_case(n, H, d, dv, channel, spread=1.0)
    case[4].fill_(center)
    case[5].zero_()
    qkv, beta, al, A_log, dt, _ = (x.double() for x in case)
    q, k, v = (qkv[:, a:a + m].reshape(n, H, -1) for a, m in ((0, H * d), (H * d, H * d), (2 * H * d, H * dv)))
    unit = lambda x: x / torch.sqrt((x ** 2).sum(-1, keepdim=True) + 1e-6)
    q, k, beta = unit(q) * d ** -0.5, unit(k), torch.sigmoid(beta)
    g = torch.exp(-torch.exp(A_log)[:, None] * torch.nn.functional.softplus(al + dt).view(n, H, -1))
    S, want = torch.zeros(H, dv, d, dtype=torch.float64, device=DEV), torch.zeros(n, H, dv, dtype=torch.float64, device=DEV)
    for t in range(n):
        S = S * g[t][:, None, :]
        S = S + (beta[t][:, None] * (v[t] - (S @ k[t][:, :, None])[..., 0]))[:, :, None] * k[t][:, None, :]
        want[t] = (S @ q[t][:, :, None])[..., 0]
    (got, state), (one, state1) = _delta_run(case, H, d, dv, channel, True), _delta_run(case, H, d, dv, channel, False)
    far = lambda x, y: float((x.double() - y).norm() / y.norm())
    assert far(got, want) < share * far(one, want)
    # (a state is the work of a few tokens where it forgets: fewer roundings to compare)
    assert far(state, S) < (share if center < -2.0 else 1.3) * far(state1, S)


def test_delta_rule_over_many_tokens_keeps_a_bounded_scratch(monkeypatch):
    """40,000 tokens of 16 heads of 128 would keep 680 MB: the room taken is the bound's, and the launches are counted."""
    from garlic_inference_b200.ops import counters, kernels
    H, Hk, d, dv, n = 16, 8, 128, 16, 40000
    qkv, ab, al = rnd(n, 2 * Hk * d + H * dv, seed=1), rnd(n, 2 * H, seed=2), rnd(n, H * d, seed=3)
    spans = torch.tensor([[0, 0, n]], dtype=torch.int32, device=DEV)
    args = (qkv, (0, Hk * d, 2 * Hk * d), ab, (H, 0), rnd(H, seed=4), rnd(H * d, seed=5), torch.zeros(1, H * dv * d, device=DEV), spans,
            torch.zeros(n, dtype=torch.int32, device=DEV), H, Hk, d, dv, 1e-6)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    torch.cuda.reset_peak_memory_stats()
    before, launched = torch.cuda.memory_allocated(), counters.launches
    out = kernels.delta_scan(*args, channel_decay=True, decay_logits=al)
    assert torch.cuda.max_memory_allocated() - before <= out.numel() * 4 + (256 << 20) + (4 << 20)
    assert counters.launches - launched == 2 * 3
    del out


# ---- experts' products ------------------------------------------------------------------------------------------------------------
@pytest.mark.parametrize("E, K, n_out", [(4, 64, 128), (3, 72, 200), (40, 128, 96), (16, 1032, 264)])
@pytest.mark.parametrize("counts", ["even", "one", "none_first", "many"])
@pytest.mark.parametrize("unit", [None, "relu_squared", "glu"])
def test_products_of_the_experts_rows(E, K, n_out, counts, unit):
    """Experts without rows, one with all of them, parts of tiles on every side, row counts on both sides of an item's 32 and
    64 rows, against 64 bits."""
    from garlic_inference_b200.ops import kernels
    n = {"even": [3] * E, "one": [0] * (E - 1) + [70], "none_first": [0, 33, 0] + [1] * (E - 3),
         "many": [65 + 7 * (e % 3) for e in range(E)]}[counts]
    ends = torch.tensor([sum(n[:e + 1]) for e in range(E)], dtype=torch.int32, device=DEV)
    glu = kernels.glu_shape("swish", 1.7, 1.5, 1.0, 1.0) if unit == "glu" else unit
    rows = rnd(sum(n), K, seed=1, dtype=torch.bfloat16)
    w = rnd(E, n_out * (2 if unit == "glu" else 1), K, seed=2, scale=K ** -0.5, dtype=torch.bfloat16)
    got = kernels.moe_products(rows, ends, w, glu)
    at = 0
    for e in range(E):
        z = rows[at:at + n[e]].double() @ w[e].double().T
        if unit == "relu_squared":
            z = z.clamp(min=0) ** 2
        elif unit == "glu":
            g, u = z[:, :n_out].clamp(max=1.5), z[:, n_out:].clamp(-1.0, 1.0)
            z = g * torch.sigmoid(1.7 * g) * (u + 1.0)
        torch.testing.assert_close(got[at:at + n[e]].double(), z, rtol=2.0 ** -8, atol=1e-4)      # one rounding, float32 sums
        at += n[e]
    kernels.check_bounded_waits(torch.device("cuda", 0))


@pytest.mark.parametrize("unit", ["glu", "relu_squared"])
@pytest.mark.parametrize("n", [1, 2, 8, 9])
def test_routed_experts_of_few_rows_by_rows_and_by_products(unit, n, monkeypatch):
    """The part's two ways for a decode step's rows, chosen by the bytes of the pairs' matrices."""
    import garlic_inference_b200.parts.moe as moe
    from garlic_inference_b200.parts import Runtime, StepContext
    params = dict(hidden_size=64, expert_size=136, n_experts=6, top=2, expert="glu" if unit == "glu" else "two_matrix")
    w = {k: rnd(*t.shape, seed=i, scale=t.shape[-1] ** -0.5, dtype=torch.bfloat16) for i, (k, t) in enumerate(moe.RoutedExperts.wanted(params).items())}

    class Load:
        def dtype(self, *names):
            return torch.bfloat16

        def __call__(self, name, out=None):
            return w[name] if out is None else out.copy_(w[name])

    part = moe.RoutedExperts(params, Load(), Runtime(torch.bfloat16, torch.device("cuda", 0)))
    x, z = rnd(n, 64, seed=50, dtype=torch.bfloat16), torch.zeros(n, dtype=torch.int32, device=DEV)
    got = []
    for limit in (0, 1 << 40):
        monkeypatch.setattr(moe, "ROWWISE_MAX_BYTES", limit)
        got.append(part.step(x, StepContext(n, z, z, z)).double())
    torch.testing.assert_close(got[0], got[1], rtol=2e-2, atol=1e-2)       # roundings of the activation and of the pairs' results


@pytest.mark.parametrize("E, n, library, own", [(4, 128, True, True), (4, 129, True, False), (4, 128, False, True), (4, 129, False, False),
                                                (256, 20, True, True), (257, 20, True, False), (257, 20, False, False)])
def test_which_products_the_experts_run(E, n, library, own, monkeypatch):
    """Up to 64 rows an expert on average and 256 experts the package's own, also where the library has no grouped product; the
    row-by-row kernels' results either way."""
    import garlic_inference_b200.parts.moe as moe
    from garlic_inference_b200.parts import Runtime, StepContext
    params = dict(hidden_size=64, expert_size=136, n_experts=E, top=2, expert="glu")
    w = {k: rnd(*t.shape, seed=i, scale=t.shape[-1] ** -0.5, dtype=torch.bfloat16) for i, (k, t) in enumerate(moe.RoutedExperts.wanted(params).items())}

    class Load:
        def dtype(self, *names):
            return torch.bfloat16

        def __call__(self, name, out=None):
            return w[name] if out is None else out.copy_(w[name])

    part = moe.RoutedExperts(params, Load(), Runtime(torch.bfloat16, torch.device("cuda", 0)))
    if not library:
        monkeypatch.delattr(torch, "_grouped_mm")
    calls, real = [], moe.kernels.moe_products
    monkeypatch.setattr(moe.kernels, "moe_products", lambda *a: calls.append(1) or real(*a))
    x, z = rnd(n, 64, seed=50, dtype=torch.bfloat16), torch.zeros(n, dtype=torch.int32, device=DEV)
    got = part.step(x, StepContext(n, z, z, z)).double()
    assert len(calls) == (2 if own else 0)
    monkeypatch.setattr(moe, "ROWWISE_MAX_ROWS", 1 << 30)
    monkeypatch.setattr(moe, "ROWWISE_MAX_BYTES", 1 << 60)
    rowwise = part.step(x, StepContext(n, z, z, z)).double()                # a warp per matrix row, float32 sums
    torch.testing.assert_close(got, rowwise, rtol=2e-2, atol=1e-2)         # roundings of the activation and of the pairs' results


# ---- between projections and attention ----------------------------------------------------------------------------------------------
@pytest.mark.parametrize("src_dtype, dtype", [(torch.float32, torch.float32), (torch.float32, torch.bfloat16), (torch.bfloat16, torch.bfloat16)])
@pytest.mark.parametrize("d, dv, n_rot, half", [(64, 128, 0, False), (128, 64, 128, False), (128, 128, 64, True), (24, 20, 12, False),
                                                (80, 80, 72, True), (24, 20, 6, False)])
@pytest.mark.parametrize("n, bias, own", [(1, True, True), (5, False, True), (301, True, True), (7, False, False)])
def test_queries_keys_and_values_by_words_and_by_elements(src_dtype, dtype, d, dv, n_rot, half, n, bias, own):
    """The kernel that gives a head a group of lanes against the one that takes a token element by element (columns that do not
    start on words): the same bits, rotations of both layouts, sizes that are not whole groups, padding rows; and 64 bits."""
    from garlic_inference_b200.ops import kernels
    H, G, page = 5, 2, 16
    cols = H * d + (G * d + G * dv if own else 0)
    src = rnd(n, cols, seed=1, dtype=src_dtype)
    pos = (torch.arange(n, dtype=torch.int32) * 3 % 400).to(DEV)
    slots = torch.zeros(n, dtype=torch.int32, device=DEV)
    table = torch.arange(400 // page, dtype=torch.int32, device=DEV).flip(0).contiguous().view(1, -1)
    if n > 1:
        slots[n // 2] = -1
        pos[:] = torch.randperm(400, generator=torch.Generator().manual_seed(2))[:n].to(DEV)       # every token a place of its own
    freq = torch.tensor([1e4 ** (-2.0 * i / max(n_rot, 1)) for i in range(n_rot // 2)], device=DEV)
    b = rnd(cols, seed=3) if bias else None
    status = torch.zeros(1, dtype=torch.int32, device=DEV)

    def run(shift):
        wide = torch.zeros((n, -(-(cols + shift) // 4) * 4 + shift), dtype=src_dtype, device=DEV)
        wide[:, shift:shift + cols] = src
        kp = torch.zeros((400 // page, G, page, d), dtype=dtype, device=DEV)
        vp = torch.zeros((400 // page, G, page, dv), dtype=dtype, device=DEV)
        k_off, v_off = (shift + H * d, shift + H * d + G * d) if own else (-1, 0)
        q = kernels.attn_prepare(wide, shift, k_off, v_off, freq, n_rot, half, pos, slots, table if own else None, kp if own else None,
                                 vp if own else None, H, d, dtype, status, append=own, bias=b, magnitude=1.25)
        return q, kp, vp

    words, elements = run(0), run(1)
    assert all(torch.equal(x, y) for x, y in zip(words, elements)) and int(status.item()) == 0
    x = src.double() + (b.double() if bias else 0.0)
    q = x[:, :H * d].view(n, H, d)
    a = pos.double()[:, None] * freq.double()
    c, s = a.cos()[:, None] * 1.25, a.sin()[:, None] * 1.25
    u, v = (q[..., :n_rot // 2], q[..., n_rot // 2:n_rot]) if half else (q[..., 0:n_rot:2], q[..., 1:n_rot:2])
    turned = [u * c - v * s, v * c + u * s]
    want = q.clone()
    if n_rot:
        want[..., :n_rot] = torch.cat(turned, -1) if half else torch.stack(turned, -1).flatten(-2)
    tol = dict(rtol=2.0 ** -8, atol=2e-4) if dtype == torch.bfloat16 else dict(rtol=1e-5, atol=2e-4)      # float32 angles up to 400
    torch.testing.assert_close(words[0].double(), want, **tol)
    if own:
        for t in range(0, n, 11):
            if int(slots[t]) >= 0:
                at = int(pos[t])
                got = words[2][int(table[0, at // page]), :, at % page].double()
                torch.testing.assert_close(got, x[t, H * d + G * d:].view(G, dv), **tol)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("half", [False, True])
@pytest.mark.parametrize("d, dv, n_rot, H, G", [(128, 128, 128, 10, 2), (48, 64, 32, 16, 4), (64, 32, 64, 40, 8)])
def test_queries_keys_and_values_of_long_steps_have_the_bits_of_short_ones(dtype, half, d, dv, n_rot, H, G):
    """Steps that take four tokens to a block, or narrow tokens element by element, against their rows in steps of a few tokens."""
    from garlic_inference_b200.ops import kernels
    n, page, cols = 1201, 64, (H + G) * d + G * dv
    src = rnd(n, cols, seed=1, dtype=dtype)
    freq = torch.tensor([1e4 ** (-2.0 * i / n_rot) for i in range(n_rot // 2)], device=DEV)
    table = torch.arange(-(-n // page), dtype=torch.int32, device=DEV).flip(0).contiguous().view(1, -1)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)

    def run(cuts):
        kp, vp = (torch.zeros((table.numel(), G, page, w), dtype=dtype, device=DEV) for w in (d, dv))
        q = [kernels.attn_prepare(src[a:b], 0, H * d, (H + G) * d, freq, n_rot, half, torch.arange(a, b, dtype=torch.int32, device=DEV),
                                  torch.zeros(b - a, dtype=torch.int32, device=DEV), table, kp, vp, H, d, dtype, status)
             for a, b in zip(cuts, cuts[1:])]
        return torch.cat(q), kp, vp

    want = run(list(range(0, n, 200)) + [n])
    for cuts in ([0, n], [0, 383, 767, n], [0, 255, 511, n]):
        assert all(torch.equal(x, y) for x, y in zip(run(cuts), want))
    assert int(status.item()) == 0


# ---- float32 attention of many tokens --------------------------------------------------------------------------------------
@pytest.mark.parametrize("H, G, d, dv", [(8, 2, 128, 128), (6, 3, 64, 64), (3, 3, 72, 40), (16, 2, 100, 100), (4, 2, 128, 65)])
@pytest.mark.parametrize("page, lens", [(16, [301]), (64, [133, 1, 170, 2, 3]), (32, [5, 228, 61])])
@pytest.mark.parametrize("sink", [False, True])
def test_float32_attention_of_rows_that_share_their_fetches(H, G, d, dv, page, lens, sink):
    """Several heads and tokens to a block, sequences that end inside one, some behind cached tokens, rows without a sequence, a page that is
    not mapped: the bits of fewer tokens at a time, which a block a row takes; and 64 bits."""
    from garlic_inference_b200.ops import kernels
    past = [0, 100, 3, 40, 0][:len(lens)]
    per = max(p + n for p, n in zip(past, lens)) // page + 1
    table = torch.arange(len(lens) * per, dtype=torch.int32, device=DEV).view(len(lens), per).flip(0).contiguous()
    kp, vp = rnd(len(lens) * per, G, page, d, seed=1), rnd(len(lens) * per, G, page, d, seed=2)
    kp[table[0, 0].item(), 0, 1, 0] = 1e30                       # a row far above the others
    pos = torch.cat([torch.arange(p, p + n) for p, n in zip(past, lens)] + [torch.zeros(3)]).to(torch.int32).to(DEV)
    slot = torch.cat([torch.full((n,), i) for i, n in enumerate(lens)] + [torch.full((3,), -1)]).to(torch.int32).to(DEV)
    n = pos.numel()
    q, sinks = rnd(n, H, d, seed=3), rnd(H, seed=4) if sink else None
    run = lambda a, b, t, status: kernels.attention_generic(q[a:b].contiguous(), kp, vp, t, pos[a:b].contiguous(), slot[a:b].contiguous(),
                                                            d ** -0.5, 0, status, sinks=sinks, value_dim=dv)
    for t in (table, table.clone()):
        if t is not table:
            t[0, (past[0] + lens[0] - 1) // page] = -1           # the last page of the first sequence
        status = torch.zeros(2, dtype=torch.int32, device=DEV)
        got = run(0, n, t, status[:1])
        want = torch.cat([run(a, min(n, a + 18), t, status[1:]) for a in range(0, n, 18)])
        assert torch.equal(got, want) and int(status[0]) == int(status[1]) == (0 if t is table else 5)
    got = run(0, n, table, torch.zeros(1, dtype=torch.int32, device=DEV)).view(n, H, dv)
    assert not got[n - 3:].any()
    for i in range(1, len(lens)):
        for at in {sum(lens[:i]), sum(lens[:i + 1]) - 1}:
            keys, vals = (x[table[i].long()].permute(1, 0, 2, 3).reshape(G, per * page, d)[:, :int(pos[at]) + 1].double() for x in (kp, vp))
            s = torch.einsum("ghd,gkd->ghk", q[at].view(G, H // G, d).double(), keys) * d ** -0.5
            if sink:
                s = torch.cat([s, sinks.double().view(G, H // G, 1)], -1)
            w = torch.softmax(s, -1)[..., :keys.shape[1]]
            torch.testing.assert_close(got[at].view(G, H // G, dv).double(), torch.einsum("ghk,gkd->ghd", w, vals[..., :dv]), rtol=1e-5, atol=1e-5)


@pytest.mark.parametrize("H, G, d", [(4, 4, 128), (6, 3, 64), (16, 4, 100), (3, 3, 40)])
@pytest.mark.parametrize("lens", [[1] * 200, [3] * 67, [2, 5, 1, 7] * 13, [150] + [1] * 61])
@pytest.mark.parametrize("single", [False, True])
def test_float32_attention_of_neighbours_of_several_sequences(H, G, d, lens, single):
    """Single tokens and short portions side by side, rows that are none and a row beyond its table between them: the bits of a token alone."""
    from garlic_inference_b200.ops import kernels
    page, per, n = 16, 12, sum(lens)
    table = torch.arange(len(lens) * per, dtype=torch.int32, device=DEV).view(len(lens), per).flip(0).contiguous()
    kp, vp = rnd(len(lens) * per, G, page, d, seed=1), rnd(len(lens) * per, G, page, d, seed=2)
    past = [(i * 7) % 40 for i in range(len(lens))]
    pos = torch.cat([torch.arange(p, p + m) for p, m in zip(past, lens)]).to(torch.int32)
    slot = torch.cat([torch.full((m,), i) for i, m in enumerate(lens)]).to(torch.int32)
    slot[9::23], slot[n - 1], pos[n // 2] = -1, -1, per * page
    pos, slot, q = pos.to(DEV), slot.to(DEV), rnd(n, H, d, seed=3)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    got = kernels.attention_generic(q, kp, vp, table, pos, slot, d ** -0.5, 0, status, single=single)
    assert status.item() == 4
    want = torch.cat([kernels.attention_generic(q[i:i + 1].contiguous(), kp, vp, table, pos[i:i + 1].contiguous(), slot[i:i + 1].contiguous(),
                                                d ** -0.5, 0, status) for i in range(n)])
    assert torch.equal(got, want) and not got[n // 2].any() and not got[n - 1].any()


# ---- one token per sequence over latent rows ---------------------------------------------------------------------------
@pytest.mark.parametrize("row, rank, heads", [(576, 512, 32), (200, 192, 17), (72, 65, 40), (64, 33, 1), (584, 512, 20)])
@pytest.mark.parametrize("pos, n_splits", [([0], None), ([31, 32, 700, -1, 5, 63], None), ([300] * 40 + [-1], 2), ([2000, 3], 1)])
def test_latent_decode_with_slices_of_one_length(row, rank, heads, pos, n_splits):
    """Rows on both sides of the limits between the kernels, odd ranks, rows without a sequence between others, more slices than chunks and
    as many blocks as sequences, with a sink and with a window: against 64 bits."""
    from garlic_inference_b200.ops import kernels
    page, n, scale = 32, len(pos), 0.1
    per = max(pos) // page + 1
    table = torch.arange(n * per, dtype=torch.int32, device=DEV).view(n, per).flip(0).contiguous()
    q, pool = rnd(n, heads, row, seed=1, dtype=torch.bfloat16), rnd(n * per, 1, page, row, seed=2, dtype=torch.bfloat16)
    slot = torch.tensor([i if p >= 0 else -1 for i, p in enumerate(pos)], dtype=torch.int32, device=DEV)
    at = torch.tensor([max(p, 0) for p in pos], dtype=torch.int32, device=DEV)
    status, sinks = torch.zeros(1, dtype=torch.int32, device=DEV), rnd(heads, seed=3)
    for sink, window in ((None, 0), (sinks, 0), (None, 33)):
        got = kernels.latent_decode(q, pool, table, at, slot, scale, sink, rank, status, n_splits=n_splits, window=window).view(n, heads, rank).double()
        assert status.item() == 0
        for t, p in list(enumerate(pos))[::7] + [(n - 1, pos[-1])]:
            if p < 0:
                assert not got[t].any()
                continue
            keys = pool[table[t].long()].reshape(per * page, row)[max(0, p - window + 1) if window else 0:p + 1].double()
            s = q[t].double() @ keys.T * scale
            w = torch.softmax(torch.cat([s, sink.double()[:, None]], 1), -1)[:, :-1] if sink is not None else torch.softmax(s, -1)
            # the weights, their sum with them and the result are rounded to bfloat16, 2^-9 of each; the rest is float32
            bound = 1.05 * 3 * 2 ** -9 * (w @ keys[:, :rank].abs()) + 1e-5
            assert ((got[t] - w @ keys[:, :rank]).abs() <= bound).all(), (t, p)


@pytest.mark.parametrize("heads", [17, 33])
@pytest.mark.parametrize("n_splits, window", [(1, 0), (2, 0), (16, 0), (16, 40)])
def test_latent_decode_with_slices_that_hold_no_keys(heads, n_splits, window):
    """Fewer chunks of 32 rows than slices, down to a row without a sequence; the slices' buffer is left full of NaN first,
    as the allocator may hand it out."""
    from garlic_inference_b200.ops import kernels
    row, rank, page, scale = 72, 64, 16, 0.2
    pos = [0, 31, 32, 70, 200, 0]
    n, per = len(pos), 13
    table = torch.arange(n * per, dtype=torch.int32, device=DEV).view(n, per).flip(0).contiguous()
    q, pool = rnd(n, heads, row, seed=1, dtype=torch.bfloat16), rnd(n * per, 1, page, row, seed=2, dtype=torch.bfloat16)
    slot = torch.tensor(list(range(n - 1)) + [-1], dtype=torch.int32, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    buffer = torch.full((n, n_splits, heads, rank + 2), float("nan"), device=DEV)
    del buffer
    got = kernels.latent_decode(q, pool, table, torch.tensor(pos, dtype=torch.int32, device=DEV), slot, scale, None, rank, status,
                                n_splits=n_splits, window=window).view(n, heads, rank).double()
    assert status.item() == 0 and not got[-1].any()
    for t, p in enumerate(pos[:-1]):
        keys = pool[table[t].long()].reshape(per * page, row)[max(0, p - window + 1) if window else 0:p + 1].double()
        w = torch.softmax(q[t].double() @ keys.T * scale, -1)
        # the weights and the result are rounded to bfloat16, 2^-9 of each; the rest is float32
        bound = 1.1 * 2 ** -8 * (w @ keys[:, :rank].abs()) + 1e-5
        assert ((got[t] - w @ keys[:, :rank]).abs() <= bound).all()


@pytest.mark.parametrize("row, rank, heads", [(576, 512, 32), (192, 128, 16), (200, 33, 5), (584, 512, 20), (1600, 512, 4)])
@pytest.mark.parametrize("below", [(0, 1024), (1024, 2048), (0, 32), (64, 96), (0, 2048)])
@pytest.mark.parametrize("sink", [False, True])
def test_latent_decode_over_scores_of_minus_infinity(row, rank, heads, below, sink):
    """Whole chunks and whole slices of keys whose scores are below the finite weigh nothing, and leave the others' sums alone."""
    from garlic_inference_b200.ops import kernels
    page, n = 64, 2048
    pool, q = rnd(n // page, 1, page, row, seed=1, dtype=torch.bfloat16), rnd(1, heads, row, seed=2, dtype=torch.bfloat16)
    q[..., -1] = 100.0
    pool.view(n, row)[below[0]:below[1], -1] = -3e38
    table = torch.arange(n // page, dtype=torch.int32, device=DEV).view(1, -1)
    pos, slot, status = (torch.tensor([v], dtype=torch.int32, device=DEV) for v in (n - 1, 0, 0))
    sinks = rnd(heads, seed=3) if sink else None
    keys = pool.view(n, row).double()
    s = q[0].double() @ keys.T * 0.05
    s[:, below[0]:below[1]] = -math.inf
    w = torch.softmax(torch.cat([s, sinks.double()[:, None]], 1), -1)[:, :-1] if sink else torch.softmax(s, -1).nan_to_num(0.0)
    for splits in (1, 2, None):
        got = kernels.latent_decode(q, pool, table, pos, slot, 0.05, sinks, rank, status, n_splits=splits).view(heads, rank).double()
        # as in test_latent_decode_with_slices_that_hold_no_keys
        assert ((got - w @ keys[:, :rank]).abs() <= 1.1 * 2 ** -8 * (w @ keys[:, :rank].abs()) + 1e-5).all()


@pytest.mark.parametrize("row, rank, heads", [(576, 512, 3), (192, 128, 40), (584, 512, 2), (1600, 512, 1)])
@pytest.mark.parametrize("n, n_splits", [(64, None), (150, None), (256, None), (256, 1), (257, None), (257, 3), (600, None)])
def test_latent_decode_of_hundreds_of_sequences(row, rank, heads, n, n_splits):
    """Both sides of the count up to which slices are of one length: short sequences, one long one, rows that are none, and a row beyond its
    table that is told and gets zeros."""
    from garlic_inference_b200.ops import kernels
    page, per, scale = 32, 30, 0.1
    table = (torch.arange(n * per, dtype=torch.int32, device=DEV) % 997).view(n, per).flip(0).contiguous()
    q, pool = rnd(n, heads, row, seed=1, dtype=torch.bfloat16), rnd(997, 1, page, row, seed=2, dtype=torch.bfloat16)
    pos = torch.tensor([(i * 37) % 90 for i in range(n)], dtype=torch.int32)
    pos[n // 2], pos[n // 3] = 900, per * page
    slot = torch.arange(n, dtype=torch.int32)
    slot[5::11] = -1
    slot[n // 2], slot[n // 3] = n // 2, n // 3
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    got = kernels.latent_decode(q, pool, table, pos.to(DEV), slot.to(DEV), scale, None, rank, status, n_splits=n_splits).view(n, heads, rank).double()
    assert status.item() == 4
    for t in range(n):
        if slot[t] < 0 or t == n // 3:
            assert not got[t].any()
            continue
        keys = pool[table[t].long()].reshape(per * page, row)[:pos[t] + 1].double()
        w = torch.softmax(q[t].double() @ keys.T * scale, -1)
        # the weights, their sum with them and the result are rounded to bfloat16, 2^-9 of each at most: three times that of what is summed
        assert ((got[t] - w @ keys[:, :rank]).abs() <= 3.1 * 2 ** -9 * (w @ keys[:, :rank].abs()) + 1e-5).all(), t
