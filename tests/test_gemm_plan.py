"""The layout of a tensor-core launch (`wrk_matmul_plan`), over the sizes it may be asked for.  No GPU is touched."""
import itertools

import pytest

FP16, INT8, NF4 = 0, 1, 2
TOKENS = list(range(16, 272, 16)) + [17, 65, 1000]
WIDTHS = [128 * b for b in (1, 2, 3, 4, 5, 6, 7, 8, 10, 12, 13, 16, 20, 21, 32, 40, 70, 112)]
ROW_TILES = [1, 6, 16, 32, 80, 112, 512]


def _plans(wrk, kinds):
    for kind, k, n, rows in itertools.product(kinds, WIDTHS, TOKENS, ROW_TILES):
        yield (kind, k, n, rows), wrk.matmul_plan(kind, k, n, rows)


def _stale(raw, a_stages, walk):
    """Whether a dequantizing group can take a raw stage for filled while its previous use is still on its way.

    Group g takes pairs g, g + 2, ...; pair u lives in raw stage u % raw and A stage u % a_stages.  A wait on a phase's parity
    also succeeds when the barrier is two phases behind, so the group must know that pair u - raw has arrived.  It knows of
    its own earlier pairs, and through its waits for A stages that every pair up to (its last pair) - a_stages has been multiplied."""
    for u in range(raw, walk):
        own = (u - raw) % 2 == u % 2
        multiplied = u - 2 - a_stages
        if not own and multiplied < u - raw:
            return True
    return False


def test_a_raw_stage_is_never_taken_for_its_previous_use(wrk):
    assert _stale(5, 6, 6) and not _stale(5, 3, 9) and not _stale(4, 6, 6)  # the model itself
    for case, p in _plans(wrk, (INT8, NF4)):
        assert not _stale(p["raw"], p["a_stages"], p["walk"]), (case, p)


def test_stages_fit_the_memories(wrk):
    for case, p in _plans(wrk, (FP16, INT8, NF4)):
        kind, k, n, _ = case
        quantized = kind != FP16
        assert p["b_stages"] >= 2 and (not quantized or (p["raw"] >= 2 and p["a_stages"] >= 2)), (case, p)
        assert p["acc_cols"] + 64 * p["a_stages"] <= p["tmem_cols"] <= 512, (case, p)
        rings = p["b_stages"] * p["bu"] * p["n_tile"] * 128
        rings += p["raw"] * 128 * (128 if kind == INT8 else 64) + 8192 if quantized else p["b_stages"] * p["bu"] * 16384
        assert max(rings, p["n_tile"] * 512) + 1024 <= p["smem"] <= 223 * 1024, (case, p)
        assert 1 <= p["splits"] <= 8 and p["splits"] * p["walk"] * (2 if quantized else p["bu"]) * 64 >= k, (case, p)


def test_ctas_that_wait_for_each_other_do_not_share_an_sm(wrk):
    # Split K: a CTA holds its tensor memory until its cluster has met.  Two launches on one SM could then each hold what the
    # other waits for on the next, unless the SM's shared memory (228 KB, 1 KB of it the system's for each CTA) has room for one.
    for case, p in _plans(wrk, (FP16, INT8, NF4)):
        assert p["splits"] == 1 or 2 * (p["smem"] + 1024) > 228 * 1024, (case, p)


def test_sizes_that_are_no_matmul_are_refused(wrk):
    for bad in ((3, 256, 16, 1), (INT8, 100, 16, 1), (INT8, 256, 0, 1), (INT8, 256, 16, 0), (INT8, 256, 2 ** 32 - 1, 1)):
        with pytest.raises(wrk.WrkError):
            wrk.matmul_plan(*bad)
    assert wrk.matmul_plan(INT8, 4096, 2 ** 24, 2 ** 24)["splits"] == 1  # no product of them wraps
