"""Tensor-memory GEMM (matmul_mat_* with 16 or more tokens) against the CPU oracle: token counts around the
tile sizes, ragged row counts, split-K shapes (clusters of 4, 7 and 8 CTAs that add their partial tiles through
distributed shared memory), output types, activations, views, and repeated launches.  Tolerance: tests/util.py."""
import numpy as np
import pytest

from oracle import oracle
from tests.test_gpu_matmul import KINDS, _make_matrix, _run
from tests.util import assert_close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("n", [16, 31, 100, 256, 257, 600])
def test_token_counts_around_the_tiles(wrk, ctx, kind, n):
    got, want = _run(wrk, ctx, kind, 1024, 384, n, turbo=(n % 32 == 0), seed=n)
    assert_close(got, want, f"{kind} n={n}")


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("k,m,n", [(2048, 256, 64), (4096, 128, 32), (2048, 2048, 256), (512, 4099, 48), (7168, 300, 128)])
def test_split_k_and_ragged_rows(wrk, ctx, kind, k, m, n):
    # few output tiles and a long K: K is split over a cluster (4, 8, 4 with 128-token tiles, none, 7 CTAs);
    # 4099 / 300 rows: last tile ragged
    got, want = _run(wrk, ctx, kind, k, m, n, turbo=True, seed=k + m + n)
    assert_close(got, want, f"{kind} {k}x{m} n={n}")


@pytest.mark.parametrize("kind", KINDS)
def test_fp16_output_and_activation(wrk, ctx, kind):
    got, want = _run(wrk, ctx, kind, 1024, 512, 64, turbo=True, out_dt=np.float16, act=1, seed=3)  # squared relu
    assert_close(got, want, f"{kind} f16 out, squared relu")
    got, want = _run(wrk, ctx, kind, 1024, 512, 64, turbo=True, act=2, seed=4)  # tanh
    assert_close(got, want, f"{kind} tanh")


def test_repeated_split_k_launches(wrk, ctx):
    rng = np.random.default_rng(11)
    w = (rng.standard_normal((256, 2048), dtype=np.float32) * 0.02).astype(np.float16)
    mat, (okind, om, oscale) = _make_matrix(wrk, ctx, "int8", w)
    y = ctx.tensor(wrk.F32, [256, 64])
    for rep in range(3):
        x = rng.standard_normal((64, 2048), dtype=np.float32).astype(np.float16)
        ctx.run(mat.matmul_op(ctx.from_numpy(x), y, turbo=True))
        want = np.zeros((64, 256), dtype=np.float32)
        oracle.matmul(okind, om, oscale, x, want, mode=1)
        assert_close(y.numpy().reshape(64, 256), want, f"launch {rep}")
    assert ctx.device_status() == 0


def test_activation_view_with_row_stride(wrk, ctx):
    # activations taken as a z-slice of a [K, N, 3] tensor (as the v6 layer does with its five shifted inputs)
    rng = np.random.default_rng(12)
    K, M, N = 1024, 256, 64
    w = (rng.standard_normal((M, K), dtype=np.float32) * 0.02).astype(np.float16)
    mat, (okind, om, oscale) = _make_matrix(wrk, ctx, "nf4", w)
    x3 = rng.standard_normal((3, N, K), dtype=np.float32).astype(np.float16)
    t_x = ctx.from_numpy(x3)
    y = ctx.tensor(wrk.F32, [M, N])
    ctx.run(mat.matmul_op(t_x.view(z=2), y, turbo=True))
    want = np.zeros((N, M), dtype=np.float32)
    oracle.matmul(okind, om, oscale, np.ascontiguousarray(x3[2]), want, mode=1)
    assert_close(y.numpy().reshape(N, M), want, "z-slice input")


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("k,m,n", [(128, 128, 9), (384, 200, 15), (2688, 768, 33), (8064, 100, 17), (1152, 130, 250), (640, 129, 512)])
def test_odd_numbers_of_k_blocks_and_few_tokens(wrk, ctx, kind, k, m, n):
    # 1, 3, 21, 63, 9, 5 blocks of 128: quantized rows of these widths, and 9 or 15 tokens, are with the mma.sync kernel; fp16 from
    # 17 tokens on splits K into unequal parts (4 CTAs of 5 or 6 blocks, 8 of 7 or 8) and has fewer steps than ring stages
    got, want = _run(wrk, ctx, kind, k, m, n, turbo=True, seed=k + n)
    assert_close(got, want, f"{kind} {k}x{m} n={n}")
    assert ctx.device_status() == 0


def test_a_matmul_waits_for_the_op_that_writes_its_weights(wrk, ctx):
    # in a list a matmul starts before the ops in front of it have finished and fetches its weights at once, unless one of
    # them writes the weights: here the matrix is copied into place by the list itself
    rng = np.random.default_rng(13)
    K, M, N = 4096, 2048, 64
    w = (rng.standard_normal((M, K), dtype=np.float32) * 0.02).astype(np.float16)
    x = rng.standard_normal((N, K), dtype=np.float32).astype(np.float16)
    source, matrix, t_x = ctx.from_numpy(w), ctx.tensor(wrk.F16, [K, M], zeros=True), ctx.from_numpy(x)
    y = ctx.tensor(wrk.F32, [M, N])
    ops = wrk.op_list([wrk.blit(source, matrix), wrk.Matrix.fp16(matrix).matmul_op(t_x, y, turbo=True)])
    for graph in (False, True):
        matrix.load(np.zeros((M, K), dtype=np.float16))
        ctx.encode(ops, use_graph=graph).submit()
        assert_close(y.numpy().reshape(N, M), x.astype(np.float32) @ w.astype(np.float32).T, f"graph={graph}")


@pytest.mark.parametrize("kind,k,n", [("int8", 768, 65), ("int8", 768, 80), ("nf4", 896, 96), ("nf4", 768, 112)])
def test_more_pairs_than_raw_stages(wrk, ctx, kind, k, n):
    # six or seven pairs of steps through a ring that shared memory cuts to fewer stages
    got, want = _run(wrk, ctx, kind, k, 500, n, turbo=True, seed=k + n)
    assert_close(got, want, f"{kind} {k} n={n}")
    assert ctx.device_status() == 0


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("n", [4, 64])
@pytest.mark.parametrize("kind", KINDS)
def test_a_matmul_waits_for_earlier_ops_that_write_its_parts(wrk, ctx, kind, n, graph):
    # bytes, scales and code book come from the list itself, from an op that is not the one in front of the matmul; the kernel
    # between is short, so a matmul that fetched its weights at once would find the zeros that lay there
    rng = np.random.default_rng(14)
    K, M = 4096, 1024
    t_w = ctx.from_numpy((rng.standard_normal((M, K), dtype=np.float32) * 0.02).astype(np.float16))
    t_x = ctx.from_numpy(rng.standard_normal((n, K), dtype=np.float32).astype(np.float16))
    small = [ctx.tensor(wrk.F32, [64]) for _ in range(2)]
    y, want = ctx.tensor(wrk.F32, [M, n]), ctx.tensor(wrk.F32, [M, n])
    if kind == "fp16":
        w = ctx.tensor(wrk.F16, [K, M], zeros=True)
        parts, write = [w], [wrk.blit(t_w, w)]
        matmul = wrk.matmul_mat_fp16(w, t_x, y)
        ctx.run(wrk.Matrix.fp16(t_w).matmul_op(t_x, want, turbo=True))
    elif kind == "int8":
        w, mm = ctx.tensor(wrk.U8, [K, M], zeros=True), ctx.tensor(wrk.F16, [2 * K * M // 128], zeros=True)
        parts, write = [w, mm], [wrk.quantize_mat_int8(t_w, mm, w)]
        matmul = wrk.matmul_mat_int8(w, mm, t_x, y)
        ctx.run(wrk.Matrix.quant_u8(t_w).matmul_op(t_x, want, turbo=True))
    else:
        book, table = ctx.from_numpy(wrk.nf4_table()), ctx.from_numpy(wrk.nf4_table())
        w, am = ctx.tensor(wrk.U8, [K // 2, M], zeros=True), ctx.tensor(wrk.F16, [K * M // 64], zeros=True)
        parts, write = [w, am, table], [wrk.quantize_mat_nf4(t_w, book, am, w), wrk.blit(book, table)]
        matmul = wrk.matmul_mat_nf4(w, table, am, t_x, y)
        ctx.run(wrk.Matrix.quant_nf4(t_w).matmul_op(t_x, want, turbo=True))
    commands = ctx.encode(wrk.op_list(write + [wrk.blit(*small), matmul]), use_graph=graph)
    for _ in range(3):
        for t in parts:
            t.load(np.zeros_like(t.numpy()))
        commands.submit()
        assert np.array_equal(y.numpy(), want.numpy())
