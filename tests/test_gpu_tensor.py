"""The tensor-core kernels at the edges of their tiles, through the C ABI,
bit-exact against the oracle."""
import numpy as np
import pytest

import oracle as O

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

P = O.P


@pytest.fixture(scope="module")
def ctx():
    import zoda_b200
    c = zoda_b200.Context(0)
    yield c
    c.close()


@pytest.fixture(autouse=True)
def no_wait_gave_up(ctx):
    """After every test: no kernel's bounded wait ran out (zoda_ctx_check)."""
    yield
    ctx.check()


def to_dev(a: np.ndarray):
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.uint32).view(np.int32)).cuda()


def from_dev(t) -> np.ndarray:
    return t.cpu().numpy().view(np.uint32)


# boxes of 128 rows x 32 columns, units of 256 rows: one row over each, one column quad over
@pytest.mark.parametrize("rows", [256, 257, 384, 385, 511])
@pytest.mark.parametrize("cols", [4, 28, 32, 36, 4740])
def test_rlc_rows_tile_edges(ctx, rows, cols):
    rng = np.random.default_rng(rows * 10007 + cols)
    m = rng.integers(0, 1 << 32, size=(rows, cols), dtype=np.uint64)
    m[rows - 1] = (1 << 32) - 1  # every byte at its largest
    coeff = rng.integers(0, 1 << 32, size=(cols, 4), dtype=np.uint64)
    out = torch.empty((rows, 4), dtype=torch.int32, device="cuda")
    ctx.rlc_rows(to_dev(m.astype(np.uint32)), rows, cols, to_dev(coeff.astype(np.uint32)), out)
    torch.cuda.synchronize()
    assert np.array_equal(from_dev(out).astype(np.uint64), O.rlc_rows(m, coeff))


TENSOR_PLAN = dict(impl=3, sched=0, l2_promo=3, blocked=1, stagger=0, radix=16, ctas=0)


def extend_with(ctx, side, data, plan):
    out = torch.full((2 * side, data.shape[1]), -1, dtype=torch.int32, device="cuda")
    ctx.plan_set(side, plan)
    try:
        ctx.extend(to_dev(data), out, side, data.shape[1])
        torch.cuda.synchronize()
    finally:
        ctx.plan_clear()
    return from_dev(out)


# tiles of 128 or 256 columns, halves of 128: a quad on either side of each, several chunks,
# and the values at the ends of their range
@pytest.mark.parametrize("side", [1024, 2048, 4096])
@pytest.mark.parametrize("cols", [4, 124, 132, 256, 388, 1028])
def test_tensor_extension_tile_edges(ctx, side, cols):
    data = O.seeded_input(side, cols, seed=side + cols)
    data[:, 0] = P - 1
    data[:, 1] = 0
    assert np.array_equal(extend_with(ctx, side, data, TENSOR_PLAN), O.encode_rowmajor(data))


# rows past k read as zeros and rows past k + n are not written; the two limits cut the
# passes' column blocks at different places
@pytest.mark.parametrize("k,n", [(1000, 1000), (1024, 1), (513, 700), (1025, 1030), (1536, 2047), (2049, 2500)])
def test_tensor_encode_cut_rows(ctx, k, n):
    cols = 260
    side = 1 << (k - 1).bit_length()
    data = O.seeded_input(k, cols, seed=k + n)
    out = torch.full((k + n + 1, cols), -1, dtype=torch.int32, device="cuda")
    ctx.plan_set(side, TENSOR_PLAN)
    try:
        ctx.encode(to_dev(data), out, k, n, cols)
        torch.cuda.synchronize()
    finally:
        ctx.plan_clear()
    got = from_dev(out)
    assert np.array_equal(got[: k + n], O.encode_rowmajor(data, n))
    assert (got[k + n] == 0xFFFFFFFF).all()


@pytest.mark.parametrize("side,cols", [(1024, 16384), (2048, 8192)])
def test_tensor_extension_streams_and_capture(ctx, side, cols):
    """Wide squares on several streams at once (those of 2048 share the context's buffers in
    turn) and in a captured stream (where 2048 falls to the single-pass kernel). All bits
    agree."""
    data = O.seeded_input(side, cols, seed=5)
    ins = [to_dev(data) for _ in range(3)]
    outs = [torch.full((2 * side, cols), -1, dtype=torch.int32, device="cuda") for _ in range(4)]
    streams = [torch.cuda.Stream() for _ in range(3)]
    torch.cuda.synchronize()
    for _ in range(3):
        for i, s in enumerate(streams):
            ctx.extend(ins[i], outs[i], side, cols, stream=s)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        ctx.extend(ins[0], outs[3], side, cols)
    g.replay()
    torch.cuda.synchronize()
    want = O.encode_rowmajor(data[:, :512])
    assert np.array_equal(from_dev(outs[0][:, :512]), want)
    for o in outs[1:]:
        assert torch.equal(o, outs[0])


def test_tensor_wait_runs_out_and_the_context_survives():
    """A launch told to wait for more finished tiles than a chunk has
    (ZODA_FAULT_PIPE_WAIT): the bounded waits run out, every role of every CTA ends, the
    context reports it once and the next launch is bit-exact. No GPU fault."""
    import zoda_b200
    c = zoda_b200.Context(0)
    side, cols = 2048, 1024
    try:
        data = O.seeded_input(side, cols, seed=17)
        c.plan_set(side, TENSOR_PLAN)
        out = torch.empty((2 * side, cols), dtype=torch.int32, device="cuda")
        c.inject_fault(2)
        c.extend(to_dev(data), out, side, cols)
        with pytest.raises(zoda_b200.ZodaError) as e:
            c.check()
        assert e.value.status == 6
        c.extend(to_dev(data), out, side, cols)
        c.check()
        assert np.array_equal(from_dev(out), O.encode_rowmajor(data))
    finally:
        c.close()


# the decoder's two maps there: codewords of 2048 rows from 6144 columns on, of 4096 rows
# at any width; a ragged width, and one past the scratch's column chunk
@pytest.mark.parametrize("k,cols", [(1024, 6148), (1024, 33000), (2048, 4), (2048, 132)])
def test_tensor_recover(ctx, k, cols):
    data = torch.randint(0, P, (k, cols), dtype=torch.int32, device="cuda",
                         generator=torch.Generator(device="cuda").manual_seed(k + cols))
    code = torch.empty((2 * k, cols), dtype=torch.int32, device="cuda")
    ctx.extend(data, code, k, cols)
    rng = np.random.default_rng(k * cols)
    known = np.sort(rng.permutation(2 * k)[:k])
    known[0] = 0  # the first and the last row among them
    known[-1] = 2 * k - 1
    lost = np.setdiff1d(np.arange(2 * k), known)
    code[torch.from_numpy(lost).cuda()] = -1  # garbage: 2^32 - 1
    out = torch.full((k, cols), -1, dtype=torch.int32, device="cuda")
    ctx.recover(code, known.tolist(), k, cols, out)
    torch.cuda.synchronize()
    assert torch.equal(out, data)


# every coset of a lower rate as a map of its own, coset 0 copied on the way: n_k = 1024, 2048
# and 4096, rates 1/4 and 1/8, rows cut in the middle of a coset
@pytest.mark.parametrize("k,n", [(1000, 3000), (1024, 3072), (600, 2500), (1024, 7000), (2000, 4500), (4000, 9000)])
def test_tensor_encode_cosets(ctx, k, n):
    cols = 6148 if 1024 < k <= 2048 else 36
    data = O.seeded_input(k, cols, seed=k + n)
    out = torch.full((k + n + 1, cols), -1, dtype=torch.int32, device="cuda")
    ctx.encode(to_dev(data), out, k, n, cols)
    torch.cuda.synchronize()
    got = from_dev(out)
    w = 36
    assert np.array_equal(got[: k + n, :w], O.encode_rowmajor(np.ascontiguousarray(data[:, :w]), n))
    assert np.array_equal(got[: k + n, -w:], O.encode_rowmajor(np.ascontiguousarray(data[:, -w:]), n))
    assert (got[k + n] == 0xFFFFFFFF).all()


# one product a tile of 128 columns: a quad on either side of the tile and of a warp, several
# tiles a CTA, cut rows
@pytest.mark.parametrize("k,n", [(32, 32), (64, 64), (20, 30), (33, 40), (50, 14), (64, 1)])
@pytest.mark.parametrize("cols", [4, 28, 124, 132, 40004])
def test_tensor_small_sides(ctx, k, n, cols):
    data = O.seeded_input(k, cols, seed=k * n + cols)
    data[:, 0] = P - 1
    data[:, 1] = 0
    out = torch.full((k + n + 1, cols), -1, dtype=torch.int32, device="cuda")
    ctx.encode(to_dev(data), out, k, n, cols)
    torch.cuda.synchronize()
    got = from_dev(out)
    assert np.array_equal(got[: k + n], O.encode_rowmajor(data, n))
    assert (got[k + n] == 0xFFFFFFFF).all()


# wide squares of side 1024 leave the queue at 16384 columns; one launch, two chains, with
# and without a queue beside them, and a plan that keeps them in the queue
@pytest.mark.parametrize("shapes,plan", [
    ([(1024, 16384)], None),
    ([(1024, 16388), (1024, 16404)], None),
    ([(1024, 16384), (1024, 16380), (512, 68), (64, 132)], None),
    ([(2048, 36), (1024, 16412), (1024, 16384), (1024, 16388), (32, 4)], None),
    ([(2048, 6148), (2048, 6140), (1024, 16388), (128, 20)], None),
    ([(2048, 6144)], None),
    ([(1024, 16388), (256, 36)], dict(impl=2, sched=0, l2_promo=3, blocked=0, stagger=1, radix=16, ctas=0)),
])
def test_batch_wide_squares(ctx, shapes, plan):
    import zoda_b200
    rng = np.random.default_rng(len(shapes) * 31 + shapes[0][1])
    sq = []
    for k, cols in shapes:
        d = rng.integers(0, P, size=(k, cols), dtype=np.uint32)
        sq.append((d, to_dev(d), torch.full((2 * k, cols), -1, dtype=torch.int32, device="cuda")))
    if plan:
        ctx.plan_set(1024, plan)
    try:
        batch = zoda_b200.Batch(ctx, [(i, o, d.shape[0], d.shape[1]) for d, i, o in sq])
    finally:
        if plan:
            ctx.plan_clear()
    assert batch.elements == sum(d.size for d, _, _ in sq)
    want = [O.encode_rowmajor(d) for d, _, _ in sq]
    for _ in range(2):
        for _, _, o in sq:
            o.fill_(-1)
        batch.run()
        torch.cuda.synchronize()
        for (d, _, o), w in zip(sq, want):
            assert np.array_equal(from_dev(o), w), d.shape
    batch.close()


# the same squares through the serving loop: launches of their own beside a queue, and alone
@pytest.mark.parametrize("shapes", [[(1024, 16388), (2048, 6148), (64, 132), (1024, 64)], [(2048, 6144)]])
def test_server_wide_squares(ctx, shapes):
    import zoda_b200
    rng = np.random.default_rng(len(shapes))
    data = [rng.integers(0, P, size=s, dtype=np.uint32) for s in shapes]
    dev = [to_dev(d) for d in data]
    torch.cuda.synchronize()
    srv = zoda_b200.Server(ctx, budget_bytes=1 << 30)
    try:
        ids = [srv.submit(x, d.shape[0], d.shape[1]) for x, d in zip(dev, data)]
        for i, d in zip(ids, data):
            r = srv.wait(i)
            assert r.status == 0
            out = torch.empty((2 * d.shape[0], d.shape[1]), dtype=torch.int32, device="cuda")
            torch.cuda.synchronize()
            zoda_b200.device_copy(out, r.d_out, out.numel() * 4)
            assert np.array_equal(from_dev(out), O.encode_rowmajor(d)), d.shape
            srv.release(i)
    finally:
        srv.close()


# encodes on either side of the widths where their route changes: 512 columns (cosets 256), and one round
# of the single pass's tiles of 8 columns (4096) or three of 16 (2048)
@pytest.mark.parametrize("over", [False, True])
@pytest.mark.parametrize("k,n,fixed,per_sm", [(2100, 2000, 512, 0), (2100, 2000, 0, 8), (2100, 9000, 256, 0),
                                              (2100, 9000, 0, 8), (1100, 1000, 0, 48)])
def test_tensor_encode_route_edges(ctx, k, n, fixed, per_sm, over):
    cols = fixed + per_sm * torch.cuda.get_device_properties(0).multi_processor_count + 4 * over
    data = O.seeded_input(k, cols, seed=k + cols)
    out = torch.full((k + n, cols), -1, dtype=torch.int32, device="cuda")
    ctx.encode(to_dev(data), out, k, n, cols)
    torch.cuda.synchronize()
    for c0 in (0, cols - 20):
        want = O.encode_rowmajor(np.ascontiguousarray(data[:, c0:c0 + 20]), n)
        assert np.array_equal(from_dev(out[:, c0:c0 + 20]), want)


# the decoder on either side of the widths where its route changes: codewords of 2048 rows at
# 6144 columns, of 4096 rows at 256 and at one round of the fused pass's tiles of 8 columns
@pytest.mark.parametrize("over", [False, True])
@pytest.mark.parametrize("k,fixed,per_sm", [(1024, 6140, 0), (2048, 256, 0), (2048, 0, 8)])
def test_recover_route_edges(ctx, k, fixed, per_sm, over):
    cols = fixed + per_sm * torch.cuda.get_device_properties(0).multi_processor_count + 4 * over
    test_tensor_recover(ctx, k, cols)
