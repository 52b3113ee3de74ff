"""What a step looks like to the parts, checked on the CPU: the attention mixer's cut of the rows into query runs,
and the one copy that carries the step's int32 arrays (every array on a 16-byte boundary)."""
import numpy as np
import torch

from garlic_inference_b200.engine.step import _Staging
from garlic_inference_b200.parts import StepShape
from garlic_inference_b200.parts.attention import query_runs


def _shape(lens, past, slots=None):
    starts, row = [], 0
    for n in lens:
        starts.append(row)
        row += n
    return StepShape(slots or list(range(len(lens))), starts, list(lens), list(past), all(n == 1 for n in lens))


def test_query_runs_cover_every_row_once_and_never_cross_a_sequence():
    lens, past = [1, 37, 150, 64, 3, 129, 128, 200], [0, 10, 0, 64, 500, 1, 128, 77]
    shape = _shape(lens, past, slots=[5, 2, 9, 0, 1, 7, 3, 4])
    for rows in (64, 128, 16):
        runs = query_runs(shape, rows)
        assert runs.dtype == np.int32 and runs.shape[1] == 4
        covered = np.zeros(sum(lens), dtype=int)
        for slot, row0, n, pos0 in runs.tolist():
            i = shape.seq_slots.index(slot)
            assert 1 <= n <= rows
            assert shape.seq_starts[i] <= row0 and row0 + n <= shape.seq_starts[i] + lens[i], "a run crosses a sequence"
            assert pos0 == past[i] + (row0 - shape.seq_starts[i]), "the run's first position follows from its first row"
            covered[row0:row0 + n] += 1
        assert (covered == 1).all(), "every row in exactly one run"
        assert len(runs) == sum(-(-n // rows) for n in lens)
        keys = [p + n for _, _, n, p in runs.tolist()]
        assert keys == sorted(keys, reverse=True), "the runs with the most keys to walk come first"
    assert query_runs(_shape([], []), 64).shape == (0, 4)


def test_one_copy_carries_the_steps_arrays_each_on_a_16_byte_boundary():
    st = _Staging(torch.device("cpu"))
    arrays = [np.arange(5, dtype=np.int32), np.arange(12, dtype=np.int32).reshape(3, 4).reshape(-1),
              np.zeros(0, dtype=np.int32), np.arange(7, dtype=np.int32) * 3]
    out = st.upload(arrays)
    base = st.dev.data_ptr()
    for a, t in zip(arrays, out):
        assert t.dtype == torch.int32 and t.numel() == a.size and t.tolist() == a.tolist()
        assert (t.data_ptr() - base) % 16 == 0
    assert st.bytes_uploaded == 4 * (8 + 12 + 0 + 8)          # sizes rounded up to whole 16-byte pieces
    again = st.upload([np.arange(3, dtype=np.int32)])           # the buffers are used again
    assert again[0].tolist() == [0, 1, 2] and again[0].data_ptr() == base
    big = st.upload([np.arange(5000, dtype=np.int32)])          # and grow when a step needs more
    assert big[0].numel() == 5000 and st.capacity >= 5000 and int(big[0][-1]) == 4999


def test_mean_key_tiles_count_what_every_run_of_queries_walks():
    from garlic_inference_b200.parts.attention import _key_tiles
    shape = _shape([1, 37, 150, 64, 3, 129, 128, 700], [0, 10, 0, 64, 500, 1, 128, 77])
    for window, chunk, keep in [(0, 0, 0), (70, 0, 0), (33, 0, 70), (0, 100, 0), (1, 0, 0)]:
        walked = []
        for _, _, n, p in query_runs(shape, 128).tolist():
            first = max(0, p - window + 1) if window else 0
            if chunk:
                first = max(first, p // chunk * chunk)
            tiles = set(range(first // 64, (p + n - 1) // 64 + 1)) | set(range(min(-(-keep // 64), first // 64)))
            walked.append(len(tiles))
        tiles, runs = _key_tiles(shape, window, chunk, keep)
        assert runs == len(walked) and abs(tiles - sum(walked) / runs) < 1e-9
    assert len(shape.notes) == 5, "worked out once for each mask"
    assert _key_tiles(_shape([], []), 0, 0, 0) == (0.0, 0)


def test_queries_that_see_few_keys_keep_the_mma_sync_prompt_kernel():
    """At heads of 64, two maps or values of another size; heads of 128 always had the tcgen05 kernel."""
    from types import SimpleNamespace
    from garlic_inference_b200.ops import kernels
    from garlic_inference_b200.parts.attention import GQAAttention
    from garlic_inference_b200.parts.masked_attention import MaskedAttention
    kv = SimpleNamespace(page_size=64)
    base = dict(rt=SimpleNamespace(dtype=torch.bfloat16), window=0)
    gqa = lambda d: SimpleNamespace(d=d, n_q=32, **base)
    masked = lambda d, dv, maps, bias=None: SimpleNamespace(
        d=d, dv=dv, maps=maps, H=16, dist_bias=bias, pool=0, output_gate=False, chunk=0, keep_first=0,
        _tensor_cores=lambda: kernels.mma_attention_takes(torch.bfloat16, d, dv), **base)
    bias = torch.zeros(100, 16)
    one, two, far = _shape([3] * 300, [30] * 300), _shape([60] * 40, [60] * 40), _shape([64], [2000])
    for shape, want64, other in ((one, 64, 64), (two, 64, 128), (far, 128, 128)):
        assert GQAAttention._run_rows(gqa(64), kv, shape) == want64 and GQAAttention._run_rows(gqa(128), kv, shape) == 128
        assert MaskedAttention._run_rows(masked(64, 64, 1), kv, shape) == want64
        for m in (masked(64, 128, 2), masked(128, 64, 1), masked(128, 128, 1, bias), masked(128, 128, 2)):
            assert MaskedAttention._run_rows(m, kv, shape) == other
        assert MaskedAttention._run_rows(masked(128, 128, 1), kv, shape) == 128
    alone = _shape([100], [0])                                # two tiles, but one run: a few blocks
    assert MaskedAttention._run_rows(masked(128, 64, 1), kv, alone) == 64 and GQAAttention._run_rows(gqa(64), kv, alone) == 64
    assert GQAAttention._run_rows(gqa(64), kv) == MaskedAttention._run_rows(masked(64, 128, 2), kv) == 128
    windowed = SimpleNamespace(**{**vars(gqa(64)), "window": 40})
    assert GQAAttention._run_rows(windowed, kv, far) == 128   # positions 1,961 to 2,063: tiles 30 to 32
    assert GQAAttention._run_rows(windowed, kv, _shape([20], [2000])) == 64      # up to 2,019: two tiles of a long sequence


def test_slices_of_a_latent_decode_step():
    from garlic_inference_b200.ops.kernels import latent_decode_slices
    assert [latent_decode_slices(n, 32) for n in (1, 16, 32, 33, 64, 256, 1000)] == [16, 16, 10, 7, 4, 1, 1]
    assert [latent_decode_slices(n, 128) for n in (1, 4, 8, 16)] == [16, 16, 10, 4] and latent_decode_slices(0, 8) == 16
