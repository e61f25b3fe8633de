"""Each kernel alone against plain torch arithmetic, at sizes other than the engine's tiny models:
head sizes in steps of 16, head counts and groups that are no power of two, widths and
vocabularies that are no power of two."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda:0"
DTYPES = [torch.float32, torch.bfloat16]


@pytest.fixture(scope="module")
def ops():
    import kirai_b200  # noqa: F401
    from kirai_b200.csrc import ops as module

    module.library()
    return module


def tol(dtype, scale=1.0):
    return (2e-5 if dtype == torch.float32 else 1.6e-2) * scale


def rand(*shape, dtype=torch.float32, scale=1.0, seed=0):
    generator = torch.Generator(device="cpu").manual_seed(seed + sum(shape))
    return (torch.randn(*shape, generator=generator) * scale).to(dtype).to(DEV)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("vocab,hidden", [(1000, 72), (257, 200), (130, 4104)])
def test_embedding(ops, dtype, vocab, hidden):
    table = rand(vocab, hidden, dtype=dtype)
    ids = torch.tensor([0, vocab - 1, 5, 5, 17], dtype=torch.int32, device=DEV)
    out = ops.embedding(table, ids)
    assert out.dtype == torch.float32 and torch.equal(out, table.float()[ids.long()])
    ops.embedding(table, torch.tensor([vocab], dtype=torch.int32, device=DEV))
    with pytest.raises(ops.KernelError):
        ops.check_device_errors(torch.device(DEV))
    if dtype == torch.bfloat16:  # the gather from the tensor-core product's box layout
        boxes = ops.tile_weight(table)
        assert torch.equal(ops.embedding(boxes, ids), out)
        ops.embedding(boxes, torch.tensor([-1], dtype=torch.int32, device=DEV))
        with pytest.raises(ops.KernelError):
            ops.check_device_errors(torch.device(DEV))


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("rows,hidden,eps", [(7, 200, 1e-5), (33, 4104, 1e-6), (1, 48, 0.0)])
def test_add_rmsnorm(ops, dtype, rows, hidden, eps):
    resid = rand(rows, hidden, scale=2.0)
    delta = rand(rows, hidden, dtype=dtype, seed=1)
    weight = 1.0 + 0.1 * rand(hidden, seed=2)
    expected_sum = resid + delta.float()
    expected = expected_sum * torch.rsqrt((expected_sum ** 2).mean(-1, keepdim=True) + eps) * weight
    stream = resid.clone()
    out = ops.add_rmsnorm(stream, delta, weight, eps, dtype)
    assert torch.allclose(stream, expected_sum, atol=1e-6)
    assert float((out.float() - expected).abs().max()) <= tol(dtype, float(expected.abs().max()))
    # chosen rows only: the stream stays as it is
    index = torch.tensor([rows - 1, 0], dtype=torch.int32, device=DEV)
    stream2 = resid.clone()
    out_rows, summed = ops.add_rmsnorm(stream2, delta, weight, eps, dtype, row_index=index)
    assert torch.equal(stream2, resid) and torch.allclose(summed, expected_sum[index.long()], atol=1e-6)
    assert float((out_rows.float() - expected[index.long()]).abs().max()) <= tol(dtype, float(expected.abs().max()))
    zero = ops.add_rmsnorm(torch.zeros(2, hidden, device=DEV), None, weight, 0.0, dtype)
    assert torch.equal(zero.float(), torch.zeros(2, hidden, device=DEV))  # mean + eps == 0 gives scale 0


def rope_reference(x, positions, inv_freq, rotary_dim):
    half = rotary_dim // 2
    angle = positions.float()[:, None] * inv_freq[None, :]
    cos, sin = torch.cos(angle.double()).float()[:, None, :], torch.sin(angle.double()).float()[:, None, :]
    out = x.clone().float()
    first, second = x[..., :half].float(), x[..., half:rotary_dim].float()
    out[..., :half] = first * cos - second * sin
    out[..., half:rotary_dim] = second * cos + first * sin
    return out


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("heads,width,rotary", [(3, 48, 48), (5, 80, 32), (2, 256, 256)])
def test_rope_and_head_rmsnorm(ops, dtype, heads, width, rotary):
    rows = 19
    buffer = rand(rows, heads * width + 24, dtype=dtype)  # heads live inside a wider row
    x = buffer[:, : heads * width].unflatten(1, (heads, width))
    positions = torch.tensor([0, 1, 2, 3, 100, 4095, 40959, 7, 8, 9, 10, 11, 12, 13, 14, 15, 16, 17, 31], dtype=torch.int32, device=DEV)
    inv_freq = torch.pow(torch.tensor(1e6), -(2.0 * torch.arange(rotary // 2)) / rotary).to(DEV)
    expected = rope_reference(x, positions, inv_freq, rotary)
    before_tail = buffer[:, heads * width :].clone()
    ops.rope_(x, positions, inv_freq, rotary)
    assert float((x.float() - expected).abs().max()) <= tol(dtype, float(expected.abs().max()))
    assert torch.equal(buffer[:, heads * width :], before_tail)
    weight = 1.0 + 0.1 * rand(width, seed=5)
    y = x.clone()
    expected = y.float() * torch.rsqrt((y.float() ** 2).mean(-1, keepdim=True) + 1e-5) * weight
    ops.head_rmsnorm_(y, weight, 1e-5)
    assert float((y.float() - expected).abs().max()) <= tol(dtype, float(expected.abs().max()))


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("rows,inter", [(5, 200), (130, 1000)])
def test_swiglu(ops, dtype, rows, inter):
    gate_up = rand(rows, 2 * inter, dtype=dtype, scale=3.0)
    g, u = gate_up[:, :inter].float(), gate_up[:, inter:].float()
    expected = g / (1.0 + torch.exp(-g)) * u
    out = ops.swiglu(gate_up)
    assert float((out.float() - expected).abs().max()) <= tol(dtype, float(expected.abs().max()))


@pytest.mark.parametrize("m,n,k", [(1, 40, 24), (7, 130, 200), (70, 257, 72), (129, 64, 1000)])
def test_linear_plain_float32_is_exact_enough(ops, m, n, k):
    x, w = rand(m, k), rand(n, k, seed=3)
    expected = (x.double() @ w.double().T).float()
    out = ops.linear_plain(x, w)
    assert float((out - expected).abs().max()) <= 1e-5 * math.sqrt(k)


@pytest.mark.parametrize("m", [1, 2, 3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("n,k", [(1, 4), (33, 124), (31, 128), (40, 512), (9, 516), (130, 1000), (7, 4100), (1003, 2560)])
def test_linear_float32_of_few_rows(ops, m, n, k):
    """Edges of the 128-column pieces, of four warps' shares of K and of a block's rows; rows of a wider matrix."""
    x, w = rand(m, k + 8)[:, 4 : 4 + k], rand(n, k, seed=3)
    expected = x.double() @ w.double().T
    out = ops.linear(x, w)
    # every rounding of a sum of k products is at most 2^-24 of the running sum of sizes, and no sum is longer than
    # k / 32 + 16 steps (a lane's share of K, the butterfly, the warps)
    bound = (k / 32 + 16) * 2.0 ** -24 * (x.abs().double() @ w.abs().double().T)
    assert bool(((out.double() - expected).abs() <= bound).all())
    assert torch.equal(out, ops.linear_f32_rows(x, w))
    plain = ops.linear(rand(m, k + 9)[:, 1 : 1 + k], w)  # rows that are not on 16-byte boundaries: the plain kernel
    assert torch.equal(plain, ops.linear_plain(rand(m, k + 9)[:, 1 : 1 + k], w))
    x[0, 0] = float("inf")
    assert torch.equal(ops.linear(x, w)[0].isinf(), w[:, 0] != 0)


@pytest.mark.parametrize("m,n,k", [(1, 1, 4), (9, 130, 36), (32, 128, 32), (33, 127, 64), (64, 256, 96), (65, 129, 100),
                                   (128, 130, 516), (193, 300, 1028), (400, 257, 2600)])
def test_linear_float32_on_tensor_cores(ops, m, n, k):
    """Edges of the tiles (32 to 192 rows, 128 columns, 32 values of K), every cut; rows of a wider matrix."""
    x, w = rand(m, k + 8)[:, 4 : 4 + k], rand(n, k, seed=3)
    expected = x.double() @ w.double().T
    # a product leaves out what lies 2^-24 below it; sums of 32 values drop at most 2^-23 at each of 12 additions, and the
    # k / 32 sums and up to 8 shares of K are added with 2^-24 each
    bound = (14 * 2.0 ** -23 + (k / 32 + 8) * 2.0 ** -24) * (x.abs().double() @ w.abs().double().T)
    for tile_rows in (0, 32, 64, 128, 192):
        for splits in (1, 2, 3, 8):
            out = ops.linear_f32_tc(x, w, tile_rows, splits)
            assert bool(((out.double() - expected).abs() <= bound).all()), (tile_rows, splits)
    ops.check_device_errors(torch.device(DEV))
    if m > 8:
        assert torch.equal(ops.linear(x, w), ops.linear_f32_tc(x, w))
    # values that are not finite, and such as the sum of two overflows, come out as the chain of FMAs has them
    x[0, 0], x[-1, -1], w[0, k // 2] = float("inf"), float("nan"), 3e38
    plain = ops.linear_plain(x, w)
    for splits in (1, 2):
        out = ops.linear_f32_tc(x, w, 32, splits)
        assert torch.equal(out.isnan(), plain.isnan()) and torch.equal(out[out.isinf()], plain[plain.isinf()])
    with pytest.raises(AssertionError):
        ops.linear_f32_tc(rand(m, k + 9)[:, 1 : 1 + k], w)


# products whose tiles fill whole rounds of 148 SMs and a little of another: two launches (192, 128 and 32 rows a tile), the second
# with a part of a tile of columns, K split, a part of a block of K
@pytest.mark.parametrize("m,n,k", [(515, 19456, 516), (576, 6400 + 60, 1028), (128, 19200, 700), (30, 38400 + 4, 260)])
def test_linear_float32_in_whole_rounds_and_a_rest(ops, m, n, k):
    x, w = rand(m, k), rand(n, k, seed=3)
    expected = x.double() @ w.double().T
    bound = (14 * 2.0 ** -23 + (k / 32 + 8) * 2.0 ** -24) * (x.abs().double() @ w.abs().double().T)  # as above
    out = ops.linear_f32_tc(x, w)
    ops.check_device_errors(torch.device(DEV))
    assert bool(((out.double() - expected).abs() <= bound).all())
    assert torch.equal(out, ops.linear_f32_tc(x, w, constant=True))


@pytest.mark.parametrize("m", [1, 8, 40, 200])
def test_linear_float32_reads_weights_that_the_kernel_before_it_wrote(ops, m):
    """A weight made by the launch just ahead in the stream, one after the other in the same memory; and the same bits from
    weights that are said to be constant, once they are."""
    x, base = rand(m, 1024), rand(4096, 1024, seed=2)
    w = torch.empty_like(base)
    factors = [2.0 ** (i % 7 - 3) for i in range(40)]
    results = []
    for factor in factors:
        torch.mul(base, factor, out=w)
        results.append(ops.linear(x, w))
    torch.cuda.synchronize()
    want = ops.linear(x, base, constant=True)
    assert torch.equal(want, ops.linear(x, base))
    for factor, got in zip(factors, results):
        assert torch.equal(got, want * factor)  # (powers of two: every rounding is the same)
    ops.check_device_errors(torch.device(DEV))


@pytest.mark.parametrize("k", [4, 8, 16, 32])
def test_linear_float32_on_tensor_cores_leaves_out_less_than_a_rounding(ops, k):
    """Products of one sign, where what is left out cannot cancel: mantissas whose second and third cuts would be the greatest
    if a cut dropped bits, ones just under a power of two, and values spread evenly over a binade."""
    worst, full = 1.0 + 2.0 ** -7 - 2.0 ** -23, 2.0 - 2.0 ** -23
    for x, w in ((torch.full((33, k), worst), torch.full((130, k), worst)), (torch.full((33, k), full), torch.full((130, k), worst)),
                 (torch.full((33, k), full), torch.full((130, k), full)), (rand(33, k, seed=5).abs().cpu() % 1 + 1, rand(130, k, seed=6).abs().cpu() % 1 + 1)):
        x, w = x.to(DEV), w.to(DEV)
        expected = x.double() @ w.double().T
        # to nearest, the second cut is at most 2^-8 and the third 2^-17 of a value's leading bit: the products left out are within
        # 2^-24 (1 + 2^-8) of the whole; the tensor cores drop at most 2^-23 at each of the two additions of the greatest products
        # (sixteen values of K each) and 2^-8 of that at the smaller ones'
        bound = (1.01 + 2 * 2.0 * (1 + 5 * 2.0 ** -8)) * 2.0 ** -24 * expected
        assert bool(((ops.linear_f32_tc(x, w).double() - expected).abs() <= bound).all())
        # short sums, which 32-bit FMAs round less often, take those
        assert torch.equal(ops.linear(x, w), ops.linear_f32_tc(x, w) if k >= 32 else ops.linear_plain(x, w))


@pytest.mark.parametrize("k", [32, 64, 100, 2560])
def test_linear_float32_on_tensor_cores_is_nearer_than_a_chain_of_roundings(ops, k):
    """The 2-norm of the error against that of the plain kernel, over 20,000 sums: values of both signs and of one."""
    for one_sign in (False, True):
        x, w = rand(64, k, seed=7), rand(320, k, seed=8)
        x, w = (x.abs() + 1.0, w.abs() + 1.0) if one_sign else (x, w)
        expected = x.double() @ w.double().T
        error = [float((f(x, w).double() - expected).norm()) for f in (ops.linear_f32_tc, ops.linear_plain)]
        assert error[0] < error[1], (one_sign, error)


@pytest.mark.parametrize("m,n,k", [(1, 128, 64), (3, 200, 136), (16, 1000, 512), (48, 520, 1032), (64, 4096, 264),
                                   (65, 264, 192), (100, 1000, 2080), (128, 4096, 4096), (129, 520, 1032),
                                   (200, 96, 64), (256, 4096, 2112), (257, 264, 192), (300, 1000, 520), (1024, 768, 2048)])
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
def test_linear_tcgen05_against_plain(ops, m, n, k, out_dtype):
    x, w = rand(m, k, dtype=torch.bfloat16, scale=0.5), rand(n, k, dtype=torch.bfloat16, scale=0.05, seed=3)
    expected = x.float() @ w.float().T
    out = ops.linear_tcgen05(x, w, out_dtype)
    plain = ops.linear_plain(x, w, out_dtype)
    ops.check_device_errors(torch.device(DEV))
    bound = (2e-5 * math.sqrt(k) if out_dtype == torch.float32 else 1e-2) * float(expected.abs().max())
    assert float((out.float() - expected).abs().max()) <= bound
    assert float((out.float() - plain.float()).abs().max()) <= bound
    if m <= 256:  # split along K between the CTAs of a cluster (up to 64 rows: slots beside the ring; up to 256: in it)
        split = ops.linear_tcgen05(x, w, out_dtype, splits=3)
        assert float((split.float() - expected).abs().max()) <= bound
        two = ops.linear_tcgen05(x, w, out_dtype, splits=2)
        assert float((two.float() - expected).abs().max()) <= bound
    if m <= 64:
        eight = ops.linear_tcgen05(x, w, out_dtype, splits=8)  # the largest cluster
        assert float((eight.float() - expected).abs().max()) <= bound
    # a row-strided input (a slice of a wider buffer)
    wide = torch.zeros(m, k + 16, dtype=torch.bfloat16, device=DEV)
    wide[:, :k] = x
    strided = ops.linear_tcgen05(wide[:, :k], w, out_dtype)
    assert torch.equal(strided, out)
    # the same weights cut into boxes at load: the same products in the same order, bit for bit
    tiled = ops.tile_weight(w)
    assert tiled.shape == (n, k) and torch.equal(tiled.row_major(), w)
    assert torch.equal(ops.linear_tcgen05(x, tiled, out_dtype), out)
    if m <= 256:
        assert torch.equal(ops.linear_tcgen05(x, tiled, out_dtype, splits=3), split)
    assert torch.equal(ops.linear(wide[:, :k], tiled, out_dtype), out)
    ops.check_device_errors(torch.device(DEV))


@pytest.mark.parametrize("m", [1, 16, 17, 32, 33, 64, 65, 128, 200])
@pytest.mark.parametrize("splits", [2, 3, 4])
def test_split_products_of_one_block_a_cta(ops, m, splits):
    """The shortest way from a CTA's start to its first store into another CTA's shared memory: every one must have begun by then.
    The same bits each time, and the sums of 64 * splits products."""
    x, w = rand(m, 64 * splits, dtype=torch.bfloat16), rand(640, 64 * splits, dtype=torch.bfloat16, seed=3)
    tiled = ops.tile_weight(w)
    out = ops.linear_tcgen05(x, tiled, torch.float32, splits=splits)
    expected, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    assert bool(((out.double() - expected).abs() <= 64 * splits * 2.0 ** -24 * size).all())  # 32-bit sums in any order
    for _ in range(20):
        assert torch.equal(ops.linear_tcgen05(x, tiled, torch.float32, splits=splits), out)
    ops.check_device_errors(torch.device(DEV))


# tiles of the many-token kernel that the rule picks on 148 SMs: 128 and 256 rows (with a last tile of one half, or of a part of
# one), widths that cut weight boxes, columns beyond the last whole tile or box, a K that ends inside a block
@pytest.mark.parametrize("m,n,k", [(300, 2560, 64), (300, 6144, 72), (640, 2568, 136), (1100, 2560, 264), (1408, 4104, 1096),
                                   (1600, 4096, 2056), (1920, 2560, 2056), (2049, 2600, 2056), (1200, 6160, 2056)])
def test_many_token_products_of_every_tile(ops, m, n, k):
    x, w = rand(m, k, dtype=torch.bfloat16, scale=0.5), rand(n, k, dtype=torch.bfloat16, scale=0.1, seed=3)
    tiled = ops.tile_weight(w)
    # 32-bit sums of k products in another order: k roundings of 2^-24, at most, on sums of |products| (and torch's own)
    expected, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    out = ops.linear_tcgen05(x, tiled, torch.float32)
    assert bool(((out.double() - expected).abs() <= 2 * k * 2.0 ** -24 * size).all())
    assert torch.equal(out, ops.linear_tcgen05(x, w, torch.float32))
    # 16-bit results are those sums rounded once; the same bits whatever tile makes them
    assert torch.equal(ops.linear_tcgen05(x, tiled), out.bfloat16())
    assert torch.equal(ops.linear_tcgen05(x, w), out.bfloat16())
    assert torch.equal(ops.linear_relu2(x, tiled), (out.clamp(min=0.0) ** 2).bfloat16())
    if n % 16 == 0:
        gate, up = out.view(m, n // 16, 2, 8)[:, :, 0].reshape(m, -1), out.view(m, n // 16, 2, 8)[:, :, 1].reshape(m, -1)
        act = ops.linear_tcgen05(x, tiled, swiglu=True).double()
        exact = gate.double() / (1.0 + torch.exp(-gate.double())) * up.double()
        assert bool(((act - exact).abs() <= (2.0 ** -8 + 2.0 ** -18) * exact.abs() + 1e-30).all())  # one rounding to 16 bits, fast exp and division
    ops.check_device_errors(torch.device(DEV))


def test_many_token_products_take_the_tiles_tested_above(ops):
    pick = ops.library().kirai_gemm_bf16_many_tile
    shapes = test_many_token_products_of_every_tile.pytestmark[0].args[1]
    tiles = {divmod(pick(m, n, k, form), 1000) for m, n, k in shapes for form in (0, 1, 2)}
    assert {rows for rows, _ in tiles} == {1, 2} and len({width for _, width in tiles}) >= 6 and any(width % 128 for _, width in tiles)


def test_threads_whose_products_want_different_shared_memory(ops):
    """One kernel, two sizes: the smaller one, launched first by another thread, must not take from the larger one what it was
    granted before (a limit belongs to the kernel, not to a thread)."""
    from concurrent.futures import ThreadPoolExecutor

    rows = (1153, 2048)  # tiles of 256 x 144 and 256 x 240 on 148 SMs
    tiles = [divmod(ops.library().kirai_gemm_bf16_many_tile(m, 4096, 4096, 0), 1000) for m in rows]
    sizes = [ops.library().kirai_gemm_bf16_many_shared(*tile) for tile in tiles]
    assert tiles[0][0] == tiles[1][0] and sizes[0] > sizes[1]
    w = ops.tile_weight(rand(4096, 4096, dtype=torch.bfloat16, scale=0.1))
    x = [rand(m, 4096, dtype=torch.bfloat16, scale=0.5) for m in rows]
    begin = lambda: torch.ones(1, device=DEV).add_(1)  # noqa: E731  (a launch of torch's, which gives the thread its device)
    with ThreadPoolExecutor(1, initializer=begin) as first, ThreadPoolExecutor(1, initializer=begin) as second:
        wanted = first.submit(ops.linear_tcgen05, x[0], w).result()
        second.submit(ops.linear_tcgen05, x[1], w).result()
        assert torch.equal(first.submit(ops.linear_tcgen05, x[0], w).result(), wanted)
        # and at the same time
        runs = [pool.submit(lambda i=i: [ops.linear_tcgen05(x[i], w) for _ in range(50)][-1]) for i, pool in enumerate((first, second))]
        assert torch.equal(runs[0].result(), wanted) and runs[1].result().shape == (rows[1], 4096)
    ops.check_device_errors(torch.device(DEV))


def test_linear_refuses_rows_that_tma_cannot_read(ops):
    x, w = rand(4, 70, dtype=torch.bfloat16), rand(32, 70, dtype=torch.bfloat16)
    with pytest.raises(ops.KernelError):
        ops.linear_tcgen05(x, w)
    out = ops.linear(x, w)  # the product path takes the CUDA-core kernel for such a K
    expected = x.float() @ w.float().T
    assert float((out.float() - expected).abs().max()) <= 1e-2 * float(expected.abs().max())


def paged_setup(dtype, lengths, kv_heads, head_dim, page_size, seed=0):
    """Random keys and values for requests of the given lengths, scattered over shuffled pages."""
    generator = torch.Generator().manual_seed(seed)
    pages_per = [-(-n // page_size) for n in lengths]
    num_pages = sum(pages_per) + 3
    order = torch.randperm(num_pages, generator=generator).tolist()
    cache = torch.zeros(num_pages, 2, kv_heads, page_size, head_dim, dtype=dtype, device=DEV)
    width = max(pages_per)
    table = torch.full((len(lengths), width), -1, dtype=torch.int32)
    keys, values = [], []
    cursor = 0
    for r, n in enumerate(lengths):
        k = (torch.randn(n, kv_heads, head_dim, generator=generator)).to(dtype)
        v = (torch.randn(n, kv_heads, head_dim, generator=generator)).to(dtype)
        keys.append(k)
        values.append(v)
        for p in range(pages_per[r]):
            table[r, p] = order[cursor]
            cursor += 1
    return cache, table.to(DEV), keys, values


def attention_reference(q, k, v, positions, window, scale):
    """q [T, nq, d] at absolute positions of one request; k, v [n, nkv, d] all its rows."""
    nq, nkv = q.shape[1], k.shape[1]
    out = torch.zeros(q.shape, dtype=torch.float32)
    for t, pos in enumerate(positions):
        lo = 0 if not window else max(0, pos - window + 1)
        for h in range(nq):
            kv = h // (nq // nkv)
            s = (k[lo : pos + 1, kv].float() @ q[t, h].float()) * scale
            p = torch.softmax(s, dim=0)
            out[t, h] = p @ v[lo : pos + 1, kv].float()
    return out


@pytest.mark.parametrize("rows", [1, 8, 16, 23, 64])
@pytest.mark.parametrize("hidden,q_width,inter,qkv_width", [(200, 136, 328, 264), (4096, 4096, 1536, 6144), (128, 64, 16, 96)])
def test_products_held_back_and_launched_as_one_kernel(ops, monkeypatch, rows, hidden, q_width, inter, qkv_width):
    """A layer's products (output projection with the residual and the next norm, gate/up with SwiGLU, down with the
    residual and the norm, the next q/k/v) through ``chained_products`` as one persistent kernel, against the same
    calls launched one by one and against 32-bit arithmetic; twice in a row, since the kernel leaves its counters for
    its next launch."""
    eps = 1e-6
    bf = torch.bfloat16
    monkeypatch.setattr(ops, "chain_products", True)
    w_o, w_gate, w_up = rand(hidden, q_width, dtype=bf, scale=0.05), rand(inter, hidden, dtype=bf, scale=0.05, seed=1), rand(inter, hidden, dtype=bf, scale=0.05, seed=2)
    w_down, w_qkv = rand(hidden, inter, dtype=bf, scale=0.05, seed=3), rand(qkv_width, hidden, dtype=bf, scale=0.05, seed=4)
    norm1, norm2 = 1.0 + 0.1 * rand(hidden, seed=5), 1.0 + 0.1 * rand(hidden, seed=6)
    tiled = {name: ops.tile_weight(w) for name, w in (("o", w_o), ("down", w_down), ("qkv", w_qkv))}
    tiled["gate_up"] = ops.tile_weight(ops.interleave_gate_up(w_gate, w_up))
    x = rand(rows, q_width, dtype=bf, seed=7)
    stream0 = rand(rows, hidden, scale=2.0, seed=8)

    def layer(stream):
        rows1, sumsq1 = ops.linear_residual_norm(x, tiled["o"], stream, norm1)
        act = ops.linear_tcgen05(rows1, tiled["gate_up"], swiglu=True, row_scale=(sumsq1, hidden, eps))
        rows2, sumsq2 = ops.linear_residual_norm(act, tiled["down"], stream, norm2)
        return ops.linear_tcgen05(rows2, tiled["qkv"], row_scale=(sumsq2, hidden, eps))

    single_stream = stream0.clone()
    single = layer(single_stream)
    before = ops.launch_count
    for attempt in range(2):
        chained_stream = stream0.clone()
        with ops.chained_products():
            chained = layer(chained_stream)
            assert ops.chaining()
        ops.check_device_errors(torch.device(DEV))
        assert not ops.chaining()
        # 32-bit arithmetic on the same bf16 inputs, with the roundings to bf16 where the kernels round
        r1 = stream0 + x.float() @ w_o.float().T
        n1 = (r1 * norm1).to(bf).float() * torch.rsqrt((r1 ** 2).mean(-1, keepdim=True) + eps)
        gate, up = n1 @ w_gate.float().T, n1 @ w_up.float().T
        a = (gate / (1.0 + torch.exp(-gate)) * up).to(bf).float()
        r2 = r1 + a @ w_down.float().T
        n2 = (r2 * norm2).to(bf).float() * torch.rsqrt((r2 ** 2).mean(-1, keepdim=True) + eps)
        expected = n2 @ w_qkv.float().T
        scale = float(expected.abs().max())
        assert float((chained.float() - expected).abs().max()) <= tol(bf, scale)
        assert float((chained_stream - r2).abs().max()) <= tol(bf, float(r2.abs().max()))
        assert float((chained.float() - single.float()).abs().max()) <= tol(bf, scale)
        assert float((chained_stream - single_stream).abs().max()) <= tol(bf, float(r2.abs().max()))
    assert ops.launch_count - before == 2  # four products, one launch, each time


def test_products_held_back_go_out_before_any_other_kernel(ops, monkeypatch):
    """Launch order is kept: a kernel of another kind, asked for while products are held back, sees their results."""
    bf = torch.bfloat16
    monkeypatch.setattr(ops, "chain_products", True)
    w1, w2 = ops.tile_weight(rand(256, 128, dtype=bf, scale=0.1)), ops.tile_weight(rand(128, 256, dtype=bf, scale=0.1, seed=1))
    x = rand(5, 128, dtype=bf, seed=2)
    stream = torch.zeros(5, 128, device=DEV)
    with ops.chained_products():
        y = ops.linear_tcgen05(ops.linear_tcgen05(x, w1), w2)
        ops.add_into_residual(stream, y)  # not a product: the two held back are launched first
        z = ops.linear_tcgen05(y, w1)     # held back until the block ends
    expected = (x.float() @ w1.row_major().float().T).to(bf).float() @ w2.row_major().float().T
    assert float((stream - expected).abs().max()) <= tol(bf, float(expected.abs().max()))
    assert float((z.float() - y.float() @ w1.row_major().float().T).abs().max()) <= tol(bf, float(z.float().abs().max()))
    with pytest.raises(RuntimeError, match="boom"):
        with ops.chained_products():
            ops.linear_tcgen05(x, w1)
            raise RuntimeError("boom")
    assert not ops.chaining() and ops.linear_tcgen05(x, w1).shape == (5, 256)  # nothing stayed behind
    ops.check_device_errors(torch.device(DEV))


def test_a_bounded_wait_that_runs_out_is_reported_and_the_device_stays_usable(ops):
    """Every barrier wait in the kernels gives up after a number of polls, sets the device error word and lets the
    kernel return.  The self-test kernel waits for a barrier that nothing completes: the host must read "a bounded
    wait ... ran out", and the launches after it must run as if nothing had happened."""
    device = torch.device(DEV)
    assert ops.wait_selftest(device, limit=10_000, arrive=True) == 0   # the control: an answered wait is no error
    ops.check_device_errors(device)
    assert ops.wait_selftest(device, limit=10_000) == 10_000
    with pytest.raises(ops.KernelError, match="bounded wait inside a kernel ran out"):
        ops.check_device_errors(device)
    ops.check_device_errors(device)  # reading the word cleared it
    x = rand(5, 64, dtype=torch.bfloat16)
    w = rand(24, 64, dtype=torch.bfloat16, seed=1)
    out = ops.linear(x, w)  # a tensor-core product with its own barrier waits, right after
    assert float((out.float() - x.float() @ w.float().T).abs().max()) <= tol(torch.bfloat16, 8.0)
    ops.check_device_errors(device)
    with pytest.raises(ops.KernelError, match="refused"):
        ops.wait_selftest(device, limit=1 << 21)


@pytest.mark.parametrize("balanced", ["0", "1"])
@pytest.mark.parametrize("q_heads,kv_heads,head_dim,page_size,window,lengths",
                         [(32, 8, 128, 16, None, [700, 33, 512, 129, 1]), (6, 2, 64, 4, 9, [40, 7, 16]), (4, 4, 256, 64, None, [300, 65]),
                          (16, 1, 128, 8, 100, [260, 1, 17, 16, 130]), (8, 2, 128, 16, None, [4100])])
def test_decode_attention_that_prepares_its_queries_and_keys(ops, monkeypatch, balanced, q_heads, kv_heads, head_dim, page_size, window, lengths):
    """One kernel (per-head norm of q and k, rotation, the new token appended to its page, attention) against the two
    that it replaces, on the same inputs: the attention rows and every byte of the cache must be equal, with either
    way of cutting the keys (equal ranges per request, merged through a buffer; one range per
    SM), heads of 64, 128 and 256, groups of 1 to 16, a window, pages smaller and larger than a key tile."""
    from types import SimpleNamespace

    monkeypatch.setenv("KIRAI_DECODE_BALANCED", balanced)
    dtype = torch.bfloat16
    requests = len(lengths)
    cache, table, keys, values = paged_setup(dtype, lengths, kv_heads, head_dim, page_size, seed=11)
    for r, n in enumerate(lengths):  # the tokens before the new one are in the pages already
        if n > 1:
            pos = torch.arange(n - 1, dtype=torch.int32, device=DEV)
            ops.kv_write(keys[r][: n - 1].to(DEV).contiguous(), values[r][: n - 1].to(DEV).contiguous(), cache, table,
                         torch.full((n - 1,), r, dtype=torch.int32, device=DEV), pos)
    width = (q_heads + 2 * kv_heads) * head_dim
    qkv = rand(requests, width, dtype=dtype, seed=5)
    q_weight, k_weight = 1.0 + 0.1 * rand(head_dim, seed=6), 1.0 + 0.1 * rand(head_dim, seed=7)
    inv_freq = torch.pow(torch.tensor(10000.0), -torch.arange(head_dim // 2, dtype=torch.float32) * 2.0 / head_dim).to(DEV)
    positions = torch.tensor([n - 1 for n in lengths], dtype=torch.int32, device=DEV)
    context_len = torch.tensor(lengths, dtype=torch.int32, device=DEV)
    rows = torch.arange(requests, dtype=torch.int32, device=DEV)
    batch = SimpleNamespace(decode_only=True, num_requests=requests, context_len=context_len, max_context_len=max(lengths),
                            start_positions=[n - 1 for n in lengths], query_lens=[1] * requests, decode_balanced=None,
                            request_of_token=rows, positions=positions, num_decode=requests)
    scale = head_dim ** -0.5
    for weights in ((q_weight, k_weight, inv_freq), (None, None, inv_freq), (q_weight, k_weight, None)):
        qw, kw, freq = weights
        separate_cache, separate_qkv = cache.clone(), qkv.clone()
        ops.qk_norm_rope_kv_write_(separate_qkv, q_heads, kv_heads, head_dim, qw, kw, freq, 1e-6, separate_cache, table, rows, positions, True)
        q = separate_qkv[:, : q_heads * head_dim].unflatten(1, (q_heads, head_dim))
        expected = ops.paged_attention(q, separate_cache, table, batch, window, scale)
        fused_cache, fused_qkv = cache.clone(), qkv.clone()
        assert ops.decode_prepares_qk(fused_qkv, fused_cache, batch, q_heads, kv_heads, head_dim)
        crowd = SimpleNamespace(decode_only=True, num_requests=1 + ops.sm_count(torch.device(DEV)) // kv_heads)
        assert not ops.decode_prepares_qk(fused_qkv.expand(crowd.num_requests, -1) if requests == 1 else fused_qkv, fused_cache, crowd, q_heads, kv_heads, head_dim)
        got = ops.attention_decode_qk(fused_qkv, q_heads, kv_heads, head_dim, qw, kw, freq, 1e-6, fused_cache, table, batch, window, scale)
        ops.check_device_errors(torch.device(DEV))
        assert torch.equal(fused_qkv, qkv)                      # the product's rows are left as they were
        assert torch.equal(fused_cache, separate_cache)         # the same key and value rows, in the same places
        assert torch.equal(got, expected)
        assert float(got.float().abs().max()) > 0.01


def test_read_only_stream_kernel_runs_and_reports_nothing(ops):
    """The kernel that measures what a read-only stream reaches: whole 16 KB boxes only, no error word."""
    data = torch.zeros(37 * 16384, dtype=torch.uint8, device=DEV)  # fewer boxes than SMs: some CTAs have nothing to read
    ops.stream_read(data)
    ops.stream_read(torch.zeros(1000 * 16384, dtype=torch.uint8, device=DEV))
    ops.check_device_errors(torch.device(DEV))
    with pytest.raises(AssertionError):
        ops.stream_read(torch.zeros(1000, dtype=torch.uint8, device=DEV))


def test_sampler_on_the_cases_of_the_reference(ops):
    """crates/llm-sampler/src/lib.rs:222-294 through the device sampler, all rows in one launch: greedy, the first of
    equal maxima, a draw inside the nucleus, and ties inside the nucleus taken in index order."""
    from test_plain_reference import REFERENCE_TOP_P_CASES

    width = 4
    rows = [([-1.0, 0.25, 3.5, 3.0], 0.0, 1.0, 0.0, 2), ([1.0, 2.0, 2.0, -1e30], 0.0, 1.0, 0.0, 1)]
    rows += [(logits + [-1e30] * (width - len(logits)), t, p, draw, token) for logits, t, p, draw, token in REFERENCE_TOP_P_CASES]
    logits = torch.tensor([r[0] for r in rows], device=DEV)
    column = lambda i: torch.tensor([r[i] for r in rows], dtype=torch.float32, device=DEV)  # noqa: E731
    got = ops.sample_rows(logits, column(1), column(2), column(3)).tolist()
    assert got == [r[4] for r in rows]
    assert ops.argmax_rows(logits).tolist()[:2] == [2, 1]
    ops.check_device_errors(torch.device(DEV))


def test_a_row_without_a_maximum_sets_the_error_word_and_stays_in_bounds(ops):
    """All NaN or all -inf: no entry is greater than -inf.  Token 0 is written (nothing is read at a made-up index)
    and the device error word says so; rows beside it are sampled as usual."""
    logits = torch.randn(4, 300, device=DEV)
    logits[1] = float("nan")
    logits[2] = float("-inf")
    zeros, ones = torch.zeros(4, device=DEV), torch.ones(4, device=DEV)
    for temperature in (zeros, ones):
        got = ops.sample_rows(logits, temperature, ones, zeros + 0.5).tolist()
        assert got[1] == 0 and got[2] == 0 and 0 <= got[0] < 300 and 0 <= got[3] < 300
        with pytest.raises(ops.KernelError, match="no maximum"):
            ops.check_device_errors(torch.device(DEV))
    assert ops.argmax_rows(logits).tolist()[1:3] == [0, 0]
    with pytest.raises(ops.KernelError, match="no maximum"):
        ops.check_device_errors(torch.device(DEV))
    assert ops.argmax_rows(logits[:1]).tolist() == [int(logits[0].argmax())]
    ops.check_device_errors(torch.device(DEV))


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("q_heads,kv_heads,head_dim,page_size,window",
                         [(6, 2, 48, 8, None), (5, 5, 16, 4, 7), (8, 1, 128, 16, 40), (3, 1, 80, 1, None)])
def test_kv_write_and_paged_attention(ops, dtype, q_heads, kv_heads, head_dim, page_size, window):
    lengths = [37, 5, 64]
    cache, table, keys, values = paged_setup(dtype, lengths, kv_heads, head_dim, page_size)
    # write every row through the kernel, in two uneven portions per request
    for cut in (0, 1):
        rows_k, rows_v, req, pos = [], [], [], []
        for r, n in enumerate(lengths):
            lo, hi = (0, n // 3) if cut == 0 else (n // 3, n)
            rows_k.append(keys[r][lo:hi]); rows_v.append(values[r][lo:hi])
            req += [r] * (hi - lo); pos += list(range(lo, hi))
        k_rows, v_rows = torch.cat(rows_k).to(DEV).contiguous(), torch.cat(rows_v).to(DEV).contiguous()
        ops.kv_write(k_rows, v_rows, cache, table, torch.tensor(req, dtype=torch.int32, device=DEV),
                     torch.tensor(pos, dtype=torch.int32, device=DEV))
    for r, n in enumerate(lengths):
        for p in (0, n - 1):
            page = int(table[r, p // page_size])
            assert torch.equal(cache[page, 0, :, p % page_size].cpu(), keys[r][p])
            assert torch.equal(cache[page, 1, :, p % page_size].cpu(), values[r][p])
    # queries: the last 9 positions of request 0, one of request 1, the last 2 of request 2
    spans = [(0, list(range(28, 37))), (1, [4]), (2, [62, 63])]
    generator = torch.Generator().manual_seed(9)
    q = torch.randn(sum(len(s[1]) for s in spans), q_heads, head_dim, generator=generator).to(dtype)
    req = [r for r, ps in spans for _ in ps]
    pos = [p for _, ps in spans for p in ps]
    scale = head_dim ** -0.5
    out = ops.paged_attention_plain(q.to(DEV), cache, table, torch.tensor(req, dtype=torch.int32, device=DEV),
                                    torch.tensor(pos, dtype=torch.int32, device=DEV), window, scale)
    ops.check_device_errors(torch.device(DEV))
    row = 0
    for r, ps in spans:
        expected = attention_reference(q[row : row + len(ps)], keys[r], values[r], ps, window, scale)
        got = out[row : row + len(ps)].float().cpu().unflatten(1, (q_heads, head_dim))
        assert float((got - expected).abs().max()) <= tol(dtype, 4.0)
        row += len(ps)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("q_heads,kv_heads,head_dim", [(6, 2, 48), (4, 4, 16), (8, 2, 128), (2, 1, 512), (3, 1, 64), (5, 2, 256), (32, 8, 128)])
def test_fused_norm_rope_cache_write_equals_the_separate_kernels(ops, dtype, q_heads, kv_heads, head_dim):
    page_size, lengths = 8, [11, 30]
    cache_a, table, _, _ = paged_setup(dtype, lengths, kv_heads, head_dim, page_size)
    cache_b = cache_a.clone()
    rows = sum(lengths)
    qkv = rand(rows, (q_heads + 2 * kv_heads) * head_dim, dtype=dtype)
    req = torch.tensor([0] * 11 + [1] * 30, dtype=torch.int32, device=DEV)
    pos = torch.tensor(list(range(11)) + list(range(30)), dtype=torch.int32, device=DEV)
    qw, kw = 1.0 + 0.1 * rand(head_dim, seed=1), 1.0 + 0.1 * rand(head_dim, seed=2)
    inv_freq = torch.pow(torch.tensor(1e4), -(2.0 * torch.arange(head_dim // 2)) / head_dim).to(DEV)
    fused = qkv.clone()
    ops.qk_norm_rope_kv_write_(fused, q_heads, kv_heads, head_dim, qw, kw, inv_freq, 1e-6, cache_a, table, req, pos)
    separate = qkv.clone()
    nq, nkv, d = q_heads, kv_heads, head_dim
    q = separate[:, : nq * d].unflatten(1, (nq, d))
    k = separate[:, nq * d : (nq + nkv) * d].unflatten(1, (nkv, d))
    v = separate[:, (nq + nkv) * d :].unflatten(1, (nkv, d))
    ops.head_rmsnorm_(q, qw, 1e-6); ops.head_rmsnorm_(k, kw, 1e-6)
    ops.rope_(q, pos, inv_freq, d); ops.rope_(k, pos, inv_freq, d)
    ops.kv_write(k, v, cache_b, table, req, pos)
    ops.check_device_errors(torch.device(DEV))
    # the fused kernel keeps the normed value in 32-bit where the separate kernels round in between
    bound = 0.0 if dtype == torch.float32 else 0.05
    assert float((fused.float() - separate.float()).abs().max()) <= bound + 1e-6
    assert float((cache_a.float() - cache_b.float()).abs().max()) <= bound + 1e-6
    # against the formulas in 32-bit
    x = qkv.float()[:, : nq * d].unflatten(1, (nq, d))
    normed = x * torch.rsqrt((x ** 2).mean(-1, keepdim=True) + 1e-6) * qw
    expected = rope_reference(normed, pos, inv_freq, d)
    assert float((fused[:, : nq * d].float().unflatten(1, (nq, d)) - expected).abs().max()) <= tol(dtype, float(expected.abs().max()))


@pytest.mark.parametrize("vocab", [130, 257, 1000, 151936])  # 130: one block per row; the others: a row over a cluster of CTAs
def test_argmax_and_sampling(ops, vocab):
    import plain_qwen3 as plain

    generator = torch.Generator().manual_seed(vocab)
    logits = torch.randn(6, vocab, generator=generator) * 3.0
    logits[0, 5] = logits[0, 77] = 50.0        # a tie: the lower index wins
    logits[1, vocab - 1] = 60.0                # the last entry
    dev = logits.to(DEV)
    assert ops.argmax_rows(dev).tolist() == [plain.argmax_first(row) for row in logits]
    temperatures = torch.tensor([0.0, 0.7, 1.0, 1.3, 0.7, 2.0])
    top_ps = torch.tensor([1.0, 1.0, 0.9, 0.5, 0.05, 1.0])
    # Exact bookkeeping in 64-bit: the order, the running sums and the nucleus of every sampled row.
    exact = {}
    for row in range(1, 6):
        probs = torch.softmax(logits[row].double() / float(temperatures[row]), 0)
        order = torch.argsort(-probs, stable=True)
        running = torch.cumsum(probs[order], 0)
        top_p = float(top_ps[row])
        last = int(torch.searchsorted(running, torch.tensor(top_p, dtype=torch.float64))) if top_p < 1.0 else vocab - 1
        last = min(last, vocab - 1)
        rank = torch.empty(vocab, dtype=torch.long)
        rank[order] = torch.arange(vocab)
        exact[row] = (running, float(running[last]), rank)
    # 32-bit sums over a whole vocabulary carry about sqrt(V) * 2^-24 of rounding, whatever their order
    slack = 1e-4
    for draw in (0.0, 0.25, 0.5, 0.83, 0.999999):
        draws = torch.full((6,), draw)
        got = ops.sample_rows(dev, temperatures.to(DEV), top_ps.to(DEV), draws.to(DEV)).tolist()
        assert got[0] == plain.argmax_first(logits[0])
        for row in range(1, 6):
            running, total, rank = exact[row]
            place = int(rank[got[row]])
            threshold = draw * total
            before = float(running[place - 1]) if place > 0 else 0.0
            assert before - slack <= threshold <= float(running[place]) + slack, (row, draw, got[row])
            if vocab <= 1000:  # small enough that the sequential 32-bit walk of the plain implementation is exact too
                expected = plain.sample_top_p(logits[row], float(temperatures[row]), float(top_ps[row]), draw)
                assert abs(place - int(rank[expected])) <= 1, (row, draw, got[row], expected)


@pytest.mark.parametrize("vocab", [200, 1024, 4104])  # 200: one block per row; the others: a row over a cluster of CTAs
def test_sampling_among_many_equal_probabilities(ops, vocab):
    """Logits that take four values only: most entries tie with hundreds of others, inside the nucleus and at its
    edge.  Equal probabilities are ordered by index.  For every draw the sampled entry's stretch of the exact running
    sum in that order must hold the threshold, up to the rounding of 32-bit sums (ties enter the kernel's sum one by
    one, as the reference's sequential walk adds them, and a thousand additions of one small value round the same
    way each time); with top-p the entry must lie inside the exact nucleus, up to the same rounding."""
    generator = torch.Generator().manual_seed(vocab)
    logits = torch.randint(0, 4, (4, vocab), generator=generator).float()
    temperatures = torch.tensor([1.0, 0.5, 1.0, 2.0])
    top_ps = torch.tensor([1.0, 1.0, 0.6, 0.3])
    dev = logits.to(DEV)
    for draw in (0.0, 0.1, 0.37, 0.5, 0.75, 0.93, 0.999999):
        got = ops.sample_rows(dev, temperatures.to(DEV), top_ps.to(DEV), torch.full((4,), draw).to(DEV)).tolist()
        for row in range(4):
            probs = torch.softmax(logits[row].double() / float(temperatures[row]), 0)
            order = torch.argsort(-probs, stable=True)  # ties by index
            running = torch.cumsum(probs[order], 0)
            top_p = float(top_ps[row])
            last = vocab - 1 if top_p >= 1.0 else min(int(torch.searchsorted(running, torch.tensor(top_p, dtype=torch.float64))), vocab - 1)
            threshold = draw * float(running[last])
            rank = torch.empty(vocab, dtype=torch.long)
            rank[order] = torch.arange(vocab)
            place = int(rank[got[row]])
            before = float(running[place - 1]) if place > 0 else 0.0
            slack = 1e-4
            assert before - slack <= threshold <= float(running[place]) + slack, (row, draw, got[row], place)
            assert before <= float(running[last]) + slack, (row, draw, got[row], place, last)  # inside the nucleus
    ops.check_device_errors(torch.device(DEV))


@pytest.mark.parametrize("q_heads,kv_heads,head_dim,page_size,window",
                         [(6, 2, 48, 8, None), (5, 5, 16, 4, 7), (8, 2, 128, 16, 40), (32, 8, 128, 16, None),
                          (3, 1, 80, 1, None), (4, 2, 256, 64, 33), (16, 1, 64, 16, None),
                          # how the tcgen05 kernel fetches a page: whole rows in one request (head sizes 64 and 128,
                          # pages of 8 tokens and more, up to more than a tile), else panel by panel, 8 rows at most
                          (4, 2, 96, 32, None), (8, 4, 80, 4, 9), (8, 2, 128, 64, None), (4, 1, 128, 128, 50),
                          (2, 2, 64, 8, None), (2, 1, 192, 16, None)])
def test_tensor_core_attention_against_plain(ops, q_heads, kv_heads, head_dim, page_size, window):
    """Prompt portions that start in the middle of a context, and single decoded tokens, through the
    tensor-core kernels and through the plain kernel, against 32-bit arithmetic."""
    dtype = torch.bfloat16
    lengths = [150, 5, 64, 300]
    cache, table, keys, values = paged_setup(dtype, lengths, kv_heads, head_dim, page_size, seed=3)
    for r, n in enumerate(lengths):
        pos = torch.arange(n, dtype=torch.int32, device=DEV)
        ops.kv_write(keys[r].to(DEV).contiguous(), values[r].to(DEV).contiguous(), cache, table,
                     torch.full((n,), r, dtype=torch.int32, device=DEV), pos)
    scale = head_dim ** -0.5
    generator = torch.Generator().manual_seed(4)
    # mixed: the last 71 tokens of request 0, the whole of 1, one token of 2, the last 130 of 3
    spans = [(0, 150 - 71, 71), (1, 0, 5), (2, 63, 1), (3, 170, 130)]
    total = sum(s[2] for s in spans)
    q = (torch.randn(total, q_heads, head_dim, generator=generator) * 2.0).to(dtype).to(DEV)
    query_start = torch.tensor([0] + list(torch.tensor([s[2] for s in spans]).cumsum(0)), dtype=torch.int32, device=DEV)
    context_len = torch.tensor([s[1] + s[2] for s in spans], dtype=torch.int32, device=DEV)
    req = torch.tensor([i for i, s in enumerate(spans) for _ in range(s[2])], dtype=torch.int32, device=DEV)
    pos = torch.tensor([p for s in spans for p in range(s[1], s[1] + s[2])], dtype=torch.int32, device=DEV)
    # only the keys up to each request's context length count: later rows are in the pages but masked
    plain = ops.paged_attention_plain(q, cache, table, req, pos, window, scale)
    kernels = [False] + ([True] if ops.attention_prefill_takes_tcgen05(q_heads, kv_heads, head_dim, page_size) else [])
    for use_tcgen05 in kernels:  # the warp-level mma.sync kernel, and the tcgen05 kernel where it takes the shape
        fast = ops.attention_prefill(q, cache, table, query_start, context_len, max(s[2] for s in spans), window, scale,
                                     tcgen05=use_tcgen05)
        ops.check_device_errors(torch.device(DEV))
        row = 0
        for r, first, count in spans:
            expected = attention_reference(q[row : row + count].cpu(), keys[r], values[r], list(range(first, first + count)), window, scale)
            got = fast[row : row + count].float().cpu().unflatten(1, (q_heads, head_dim))
            assert float((got - expected).abs().max()) <= 2.5e-2, (use_tcgen05, r, first, count)
            row += count
        assert float((fast.float() - plain.float()).abs().max()) <= 2.5e-2
    # decode: one token per request at the end of each context, with 1, 2 and 5 splits
    if q_heads // kv_heads <= 16:
        ends = [n - 1 for n in lengths]
        qd = (torch.randn(len(lengths), q_heads, head_dim, generator=generator) * 2.0).to(dtype).to(DEV)
        ctx = torch.tensor(lengths, dtype=torch.int32, device=DEV)
        for splits in (1, 2, 5):
            got = ops.attention_decode(qd, cache, table, ctx, window, scale, splits).float().cpu().unflatten(1, (q_heads, head_dim))
            ops.check_device_errors(torch.device(DEV))
            for r, end in enumerate(ends):
                expected = attention_reference(qd[r : r + 1].cpu(), keys[r], values[r], [end], window, scale)
                assert float((got[r : r + 1] - expected).abs().max()) <= 2.5e-2, (r, splits)
        # the same with the keys of all (request, kv head) pairs cut into equal ranges: one CTA that walks through
        # every pair, a few CTAs whose borders cut pairs in two or more pieces, more CTAs than there are tiles
        for ctas in (1, 3, 7, 148, 1000):
            got = ops.attention_decode_balanced(qd, cache, table, ctx, window, scale, ctas).float().cpu().unflatten(1, (q_heads, head_dim))
            ops.check_device_errors(torch.device(DEV))
            for r, end in enumerate(ends):
                expected = attention_reference(qd[r : r + 1].cpu(), keys[r], values[r], [end], window, scale)
                assert float((got[r : r + 1] - expected).abs().max()) <= 2.5e-2, (r, ctas)


def test_prompt_attention_of_thousands_of_tokens_with_both_kernels(ops):
    """A prompt long enough that hundreds of CTAs each walk dozens of key tiles: the pipelines' barriers go through
    many phases (a wait that skipped a phase once stalled only at this size), and the two kernels must agree."""
    dtype, q_heads, kv_heads, head_dim, page_size, tokens = torch.bfloat16, 8, 2, 128, 16, 4096
    pages = tokens // page_size + 1
    generator = torch.Generator().manual_seed(9)
    cache = (torch.randn(pages, 2, kv_heads, page_size, head_dim, generator=generator) * 0.5).to(dtype).to(DEV)
    table = torch.arange(pages, dtype=torch.int32, device=DEV)[None, :].contiguous()
    q = (torch.randn(tokens, q_heads, head_dim, generator=generator)).to(dtype).to(DEV)
    qs = torch.tensor([0, tokens], dtype=torch.int32, device=DEV)
    ctx = torch.tensor([tokens], dtype=torch.int32, device=DEV)
    scale = head_dim ** -0.5
    for _ in range(3):  # the stall was a matter of timing: several launches
        fast = ops.attention_prefill(q, cache, table, qs, ctx, tokens, None, scale, tcgen05=True)
        ops.check_device_errors(torch.device(DEV))
    slow = ops.attention_prefill(q, cache, table, qs, ctx, tokens, None, scale, tcgen05=False)
    ops.check_device_errors(torch.device(DEV))
    assert float((fast.float() - slow.float()).abs().max()) <= 2.5e-2
    # a few rows against 32-bit arithmetic
    keys = cache[:, 0].permute(0, 2, 1, 3).reshape(-1, kv_heads, head_dim)[:tokens].float().cpu()
    values = cache[:, 1].permute(0, 2, 1, 3).reshape(-1, kv_heads, head_dim)[:tokens].float().cpu()
    for row in (0, 63, 64, 2047, 4095):
        expected = attention_reference(q[row : row + 1].cpu(), keys.to(dtype), values.to(dtype), [row], None, scale)
        got = fast[row : row + 1].float().cpu().unflatten(1, (q_heads, head_dim))
        assert float((got - expected).abs().max()) <= 2.5e-2, row


def test_tensor_core_attention_finds_a_far_key(ops):
    """One key among hundreds, far back and on a page edge, is made to dominate: the output must be its value."""
    dtype, q_heads, kv_heads, head_dim, page_size = torch.bfloat16, 8, 2, 128, 16
    lengths = [777]
    cache, table, keys, values = paged_setup(dtype, lengths, kv_heads, head_dim, page_size, seed=8)
    far = 16 * 3  # first row of the fourth page
    direction = torch.randn(head_dim, generator=torch.Generator().manual_seed(1))
    direction = direction / direction.norm()
    keys[0][far] = (direction * 30.0).to(dtype)
    ops.kv_write(keys[0].to(DEV).contiguous(), values[0].to(DEV).contiguous(), cache, table,
                 torch.zeros(777, dtype=torch.int32, device=DEV), torch.arange(777, dtype=torch.int32, device=DEV))
    q = (direction * 30.0).to(dtype).repeat(1, q_heads, 1).to(DEV)
    ctx = torch.tensor([777], dtype=torch.int32, device=DEV)
    for splits in (1, 4):
        out = ops.attention_decode(q, cache, table, ctx, None, head_dim ** -0.5, splits).float().cpu().unflatten(1, (q_heads, head_dim))
        for head in range(q_heads):
            assert float((out[0, head] - values[0][far, head // 4].float()).abs().max()) <= 2e-2
    for ctas in (2, 5, 148):
        out = ops.attention_decode_balanced(q, cache, table, ctx, None, head_dim ** -0.5, ctas).float().cpu().unflatten(1, (q_heads, head_dim))
        for head in range(q_heads):
            assert float((out[0, head] - values[0][far, head // 4].float()).abs().max()) <= 2e-2, ctas
    qs = torch.tensor([0, 1], dtype=torch.int32, device=DEV)
    out = ops.attention_prefill(q, cache, table, qs, ctx, 1, None, head_dim ** -0.5).float().cpu().unflatten(1, (q_heads, head_dim))
    assert float((out[0, 0] - values[0][far, 0].float()).abs().max()) <= 2e-2
    # with a window that ends one short of the far key it must vanish from the result
    out = ops.attention_decode(q, cache, table, ctx, 777 - far - 1, head_dim ** -0.5, 2).float().cpu().unflatten(1, (q_heads, head_dim))
    assert float((out[0, 0] - values[0][far, 0].float()).abs().max()) > 0.5
    out = ops.attention_decode(q, cache, table, ctx, 777 - far, head_dim ** -0.5, 2).float().cpu().unflatten(1, (q_heads, head_dim))
    assert float((out[0, 0] - values[0][far, 0].float()).abs().max()) <= 2e-2


@pytest.mark.parametrize("q_heads,kv_heads,head_dim", [(8, 2, 128), (32, 2, 64), (3, 1, 256)])
def test_decode_attention_cut_into_any_number_of_ranges(ops, q_heads, kv_heads, head_dim):
    """Every number of ranges from 2 to 18 and some beyond (more ranges than key tiles too: the empty ones must not
    count) against one range, whose result needs no merge: the merge may differ from it by rounding only."""
    dtype, page_size, length = torch.bfloat16, 16, 1500
    cache, table, keys, values = paged_setup(dtype, [length], kv_heads, head_dim, page_size, seed=21)
    ops.kv_write(keys[0].to(DEV).contiguous(), values[0].to(DEV).contiguous(), cache, table,
                 torch.zeros(length, dtype=torch.int32, device=DEV), torch.arange(length, dtype=torch.int32, device=DEV))
    q = rand(1, q_heads, head_dim, dtype=dtype, seed=22)
    ctx = torch.tensor([length], dtype=torch.int32, device=DEV)
    scale = head_dim ** -0.5
    one = ops.attention_decode(q, cache, table, ctx, None, scale, 1).float()
    plain = ops.paged_attention_plain(q, cache, table, torch.zeros(1, dtype=torch.int32, device=DEV),
                                      torch.tensor([length - 1], dtype=torch.int32, device=DEV), None, scale).float()
    assert float((one - plain).abs().max()) <= 2.5e-2
    for splits in list(range(2, 19)) + [33, 64, 100]:
        got = ops.attention_decode(q, cache, table, ctx, None, scale, splits)
        assert float((got.float() - one).abs().max()) <= 1e-2, splits
    ops.check_device_errors(q.device)


@pytest.mark.parametrize("q_heads,kv_heads,head_dim", [(8, 2, 128), (32, 2, 64), (6, 6, 48)])
def test_decode_attention_with_more_ranges_than_keys(ops, q_heads, kv_heads, head_dim):
    """Clusters of two to five CTAs of which some have no keys and come to their stores into the first CTA's shared memory at once."""
    dtype, page_size, lengths = torch.bfloat16, 16, [1, 15, 17, 40]
    cache, table, keys, values = paged_setup(dtype, lengths, kv_heads, head_dim, page_size, seed=31)
    for r, length in enumerate(lengths):
        ops.kv_write(keys[r].to(DEV).contiguous(), values[r].to(DEV).contiguous(), cache, table,
                     torch.full((length,), r, dtype=torch.int32, device=DEV), torch.arange(length, dtype=torch.int32, device=DEV))
    q = rand(len(lengths), q_heads, head_dim, dtype=dtype, seed=32)
    ctx = torch.tensor(lengths, dtype=torch.int32, device=DEV)
    one = ops.attention_decode(q, cache, table, ctx, None, head_dim ** -0.5, 1).float()
    for splits in (2, 3, 4, 5):
        got = ops.attention_decode(q, cache, table, ctx, None, head_dim ** -0.5, splits)
        # one rounding of the result and the weights to bfloat16 (2^-9 each) on values of up to about 4, as above
        assert float((got.float() - one).abs().max()) <= 1e-2, splits
        for _ in range(10):
            assert torch.equal(ops.attention_decode(q, cache, table, ctx, None, head_dim ** -0.5, splits), got), splits
    ops.check_device_errors(q.device)


@pytest.mark.parametrize("m,inter,k,splits", [(1, 128, 64, 0), (5, 200, 136, 0), (16, 1000, 512, 3), (64, 1536, 1032, 8),
                                              (65, 264, 192, 0), (128, 1536, 1032, 0), (100, 6144, 1024, 3), (250, 1536, 2048, 2),
                                              (300, 1000, 520, 0), (1024, 768, 256, 0)])
def test_linear_swiglu_epilogue(ops, m, inter, k, splits):
    x = rand(m, k, dtype=torch.bfloat16, scale=0.5)
    gate, up = rand(inter, k, dtype=torch.bfloat16, scale=0.1, seed=3), rand(inter, k, dtype=torch.bfloat16, scale=0.1, seed=4)
    weight = ops.interleave_gate_up(gate, up)
    assert torch.equal(weight[:8], gate[:8]) and torch.equal(weight[8:16], up[:8]) and torch.equal(weight[16:24], gate[8:16])
    g, u = x.float() @ gate.float().T, x.float() @ up.float().T
    expected = g / (1.0 + torch.exp(-g)) * u
    out = ops.linear_tcgen05(x, weight, splits=splits, swiglu=True)
    ops.check_device_errors(torch.device(DEV))
    assert out.shape == (m, inter)
    assert float((out.float() - expected).abs().max()) <= 1e-2 * float(expected.abs().max())
    separate = ops.swiglu(ops.linear_tcgen05(x, torch.cat([gate, up])))  # rounds gate and up to bf16 in between
    assert float((out.float() - separate.float()).abs().max()) <= 2e-2 * float(expected.abs().max())
    assert torch.equal(ops.linear_tcgen05(x, ops.tile_weight(weight), splits=splits, swiglu=True), out)
    ops.check_device_errors(torch.device(DEV))


@pytest.mark.parametrize("m,n,k,splits", [(1, 128, 64, 0), (5, 200, 136, 0), (16, 1000, 512, 3), (40, 520, 1032, 4),
                                          (64, 1536, 264, 0), (65, 264, 192, 0), (128, 4096, 1032, 3), (70, 520, 2048, 2),
                                          (256, 1024, 2048, 3), (180, 520, 520, 0), (300, 1000, 520, 0), (1024, 768, 256, 0)])
def test_linear_residual_norm_epilogue_and_row_scaled_products(ops, m, n, k, splits):
    """The product whose epilogue adds into the 32-bit stream and leaves the next norm's rows without their
    1 / rms factor, and the products that apply that factor to their result, against the formulas."""
    eps = 1e-5
    x, w = rand(m, k, dtype=torch.bfloat16, scale=0.5), rand(n, k, dtype=torch.bfloat16, scale=0.1, seed=3)
    before = rand(m, n, scale=2.0, seed=5)
    norm_weight = (1.0 + 0.3 * rand(n, seed=6)).contiguous()
    resid = before.clone()
    rows, sumsq = ops.linear_residual_norm(x, w, resid, norm_weight, splits)
    ops.check_device_errors(torch.device(DEV))
    stream = before.double() + x.double() @ w.double().T
    assert float((resid.double() - stream).abs().max()) <= 1e-5 * float(stream.abs().max())
    unscaled = stream * norm_weight.double()
    assert float((rows.double() - unscaled).abs().max()) <= 5e-3 * float(unscaled.abs().max())
    assert sumsq.shape[1] == m
    total = (stream ** 2).sum(1)
    assert float(((sumsq.double().sum(0) - total) / total).abs().max()) <= 1e-5
    again = before.clone()
    rows_tiled, sumsq_tiled = ops.linear_residual_norm(x, ops.tile_weight(w), again, norm_weight, splits)
    assert torch.equal(rows_tiled, rows) and torch.equal(sumsq_tiled, sumsq) and torch.equal(again, resid)
    # the products that follow: plain (both output types) and with the SwiGLU epilogue
    normed = unscaled * torch.rsqrt((stream ** 2).mean(1, keepdim=True) + eps)
    width = 272
    w2 = rand(width, n, dtype=torch.bfloat16, scale=0.1, seed=7)
    expected = (normed @ w2.double().T).float()
    bound = 1e-2 * float(expected.abs().max())
    for out_dtype in (torch.bfloat16, torch.float32):
        out = ops.linear_tcgen05(rows, w2, out_dtype, row_scale=(sumsq, n, eps))
        assert out.dtype == out_dtype and float((out.float() - expected).abs().max()) <= bound
    gate, up = w2[: width // 2].contiguous(), w2[width // 2:].contiguous()
    g, u = expected[:, : width // 2], expected[:, width // 2:]
    expected_act = g / (1.0 + torch.exp(-g)) * u
    act = ops.linear_tcgen05(rows, ops.interleave_gate_up(gate, up), swiglu=True, row_scale=(sumsq, n, eps))
    assert float((act.float() - expected_act).abs().max()) <= 1e-2 * float(expected_act.abs().max())
    # and against the separate kernels of the same path: add + norm, then the product
    separate_stream = before.clone()
    delta = ops.linear_tcgen05(x, w)
    separate = ops.linear_tcgen05(ops.add_rmsnorm(separate_stream, delta, norm_weight, eps, torch.bfloat16), w2, torch.float32)
    ops.check_device_errors(torch.device(DEV))
    assert float((separate - expected).abs().max()) <= 2 * bound


def test_row_scaled_product_of_a_zero_row_is_zero(ops):
    """A row whose variance plus eps is 0 gets the scale 0, as the norm kernel gives it, not a NaN."""
    m, n, k = 3, 64, 32
    x, w = torch.zeros(m, k, dtype=torch.bfloat16, device=DEV), rand(n, k, dtype=torch.bfloat16)
    resid = torch.zeros(m, n, device=DEV)
    resid[1] = 1.0
    rows, sumsq = ops.linear_residual_norm(x, w, resid, torch.ones(n, device=DEV))
    out = ops.linear_tcgen05(rows, rand(16, n, dtype=torch.bfloat16, seed=2), torch.float32, row_scale=(sumsq, n, 0.0))
    assert torch.isfinite(out).all() and float(out[0].abs().max()) == 0.0 and float(out[2].abs().max()) == 0.0
    assert float(out[1].abs().max()) > 0.0


def test_attention_with_block_tables_longer_than_the_shared_copy(ops):
    """Contexts whose block tables exceed what the kernels keep in shared memory (1,024 entries) read
    the table from global memory instead; a key near the start and one near the end must both be found."""
    dtype, q_heads, kv_heads, head_dim, page_size = torch.bfloat16, 4, 1, 64, 4
    length = 4 * 1100 + 3  # 1,101 pages
    cache, table, keys, values = paged_setup(dtype, [length], kv_heads, head_dim, page_size, seed=11)
    direction = torch.randn(head_dim, generator=torch.Generator().manual_seed(2))
    direction = direction / direction.norm()
    for marked in (5, length - 9):
        keys[0][marked] = (direction * 40.0).to(dtype)
    ops.kv_write(keys[0].to(DEV).contiguous(), values[0].to(DEV).contiguous(), cache, table,
                 torch.zeros(length, dtype=torch.int32, device=DEV), torch.arange(length, dtype=torch.int32, device=DEV))
    expected = 0.5 * (values[0][5, 0].float() + values[0][length - 9, 0].float())  # two equal scores dominate
    q = (direction * 40.0).to(dtype).repeat(1, q_heads, 1).to(DEV)
    ctx = torch.tensor([length], dtype=torch.int32, device=DEV)
    scale = head_dim ** -0.5
    for splits in (1, 3):
        out = ops.attention_decode(q, cache, table, ctx, None, scale, splits).float().cpu().unflatten(1, (q_heads, head_dim))
        assert float((out[0, 0] - expected).abs().max()) <= 3e-2, splits
    for ctas in (1, 2):  # ranges of more than 1,024 pages
        out = ops.attention_decode_balanced(q, cache, table, ctx, None, scale, ctas).float().cpu().unflatten(1, (q_heads, head_dim))
        assert float((out[0, 0] - expected).abs().max()) <= 3e-2, ctas
    qs = torch.tensor([0, 1], dtype=torch.int32, device=DEV)
    for use_tcgen05 in (False, True):
        out = ops.attention_prefill(q, cache, table, qs, ctx, 1, None, scale, tcgen05=use_tcgen05).float().cpu().unflatten(1, (q_heads, head_dim))
        assert float((out[0, 0] - expected).abs().max()) <= 3e-2, use_tcgen05
    ops.check_device_errors(torch.device(DEV))


@pytest.mark.parametrize("q_heads,kv_heads,head_dim,page_size,form",
                         [(32, 8, 128, 16, {}), (6, 2, 32, 16, {"window": 16}), (8, 1, 128, 5, {"window": 70, "keep_first": 3}),
                          (5, 5, 4, 1, {"chunk": 48}), (12, 2, 80, 7, {"softcap": 3.0}), (16, 1, 64, 64, {"sinks": True}),
                          (64, 1, 68, 16, {"window": 1}), (3, 1, 48, 8, {"chunk": 200, "sinks": True})])
def test_32_bit_attention_tiles_against_64_bit_arithmetic(ops, q_heads, kv_heads, head_dim, page_size, form):
    """Portions and single tokens through both 32-bit tile kernels.  Rows of the cache that no query may see hold NaN, and the
    last token's value is infinite: neither may reach a row that does not see it."""
    lengths, counts = [150, 5, 64, 1100], [71, 5, 1, 130]
    cache, table, keys, values = paged_setup(torch.float32, lengths, kv_heads, head_dim, page_size, seed=3)
    cache.fill_(float("nan"))
    for r, n in enumerate(lengths):
        values[r][n - 1, 0, head_dim - 1] = float("inf")
        ops.kv_write(keys[r].to(DEV).contiguous(), values[r].to(DEV).contiguous(), cache, table,
                     torch.full((n,), r, dtype=torch.int32, device=DEV), torch.arange(n, dtype=torch.int32, device=DEV))
    generator = torch.Generator().manual_seed(4)
    q = torch.randn(sum(counts), q_heads + 2, head_dim, generator=generator).to(DEV)[:, :q_heads]  # rows with a stride of their own
    scale = head_dim ** -0.5
    sinks = torch.randn(q_heads, generator=generator).to(DEV) if form.get("sinks") else None
    window, chunk, keep, cap = form.get("window"), form.get("chunk"), form.get("keep_first", 0), form.get("softcap")
    options = dict(chunk=chunk, softcap=cap, keep_first=keep, sinks=sinks)

    def expected(rows, r, positions):
        k, v = (x[r].double().to(DEV).repeat_interleave(q_heads // kv_heads, dim=1) for x in (keys, values))
        s = torch.einsum("thd,jhd->thj", rows.double(), k) * scale
        s = cap * torch.tanh(s / cap) if cap else s
        i, j = torch.tensor(positions, device=DEV)[:, None], torch.arange(len(k), device=DEV)[None, :]
        seen = (j <= i) & ((i - j < window) | (j < keep) if window else j >= i - i % chunk if chunk else True)
        s = s.masked_fill(~seen[:, None], -math.inf)
        if sinks is not None:
            s = torch.cat([s, sinks.double().view(1, -1, 1).expand(len(rows), -1, 1)], dim=-1)
        p = torch.softmax(s, dim=-1)[..., : len(k)]
        out = torch.einsum("thj,jhd->thd", p, v.nan_to_num(posinf=0.0))
        out[(seen[:, -1])[:, None] & (torch.arange(q_heads, device=DEV) < q_heads // kv_heads), head_dim - 1] = math.inf
        return out

    assert ops.attention_takes_f32_tiles(q, cache)
    # a score is a sum of up to 128 products, each rounded; weights and result follow it: (128 + 2) * 2^-24 * |q||k| scale
    # bounds a score's error by 1e-4, its usual size is a tenth of that, and the values' mean moves by as much
    bound = 3e-5
    start = torch.tensor([0] + torch.tensor(counts).cumsum(0).tolist(), dtype=torch.int32, device=DEV)
    context = torch.tensor(lengths, dtype=torch.int32, device=DEV)
    fast = ops.attention_f32_prefill(q, cache, table, start, context, max(counts), window, scale, **options).unflatten(1, (q_heads, head_dim))
    ends = torch.stack([q[int(e) - 1] for e in start[1:]])
    alone = {longest: ops.attention_f32_decode(ends, cache, table, context, longest, window, scale, **options).unflatten(1, (q_heads, head_dim))
             for longest in (1, 300, 1100)}  # one CTA, then clusters of CTAs (as many as the SMs hold)
    ops.check_device_errors(torch.device(DEV))
    for r, (n, count) in enumerate(zip(lengths, counts)):
        want = expected(q[start[r] : start[r + 1]], r, list(range(n - count, n)))
        for got, rows in [(fast[start[r] : start[r + 1]], want)] + [(a[r : r + 1], want[-1:]) for a in alone.values()]:
            finite = torch.isfinite(rows)
            assert torch.equal(torch.isfinite(got), finite)
            assert float((got.double() - rows)[finite].abs().max()) <= bound, (r, float((got.double() - rows)[finite].abs().max()))


# 32 and 8 heads: 8 CTAs for each 16 tokens.  On 148 SMs: one CTA an SM at most, two from 149 CTAs on (the order of whose second ones is
# turned), the last launch of two an SM, and one more
@pytest.mark.parametrize("tokens,before,q_heads,kv_heads,window", [(288, 0, 32, 8, None), (300, 0, 32, 8, None), (405, 0, 32, 8, None), (405, 333, 32, 8, 100),
                                                                   (592, 17, 32, 8, None), (593, 0, 32, 8, None), (1000, 0, 12, 3, None)])
def test_32_bit_attention_of_one_request_in_every_order_of_its_tiles(ops, tokens, before, q_heads, kv_heads, window):
    length, head_dim, page_size = tokens + before, 128, 16
    cache, table, keys, values = paged_setup(torch.float32, [length], kv_heads, head_dim, page_size, seed=5)
    ops.kv_write(keys[0].to(DEV).contiguous(), values[0].to(DEV).contiguous(), cache, table, torch.zeros(length, dtype=torch.int32, device=DEV),
                 torch.arange(length, dtype=torch.int32, device=DEV))
    q = rand(tokens, q_heads, head_dim, seed=6)
    start, context = (torch.tensor(v, dtype=torch.int32, device=DEV) for v in ([0, tokens], [length]))
    out = torch.full((tokens, q_heads * head_dim), float("nan"), device=DEV)
    ops.attention_f32_prefill(q, cache, table, start, context, tokens, window, head_dim ** -0.5, out=out)
    ops.check_device_errors(torch.device(DEV))
    k, v = (x[0].double().to(DEV).repeat_interleave(q_heads // kv_heads, dim=1) for x in (keys, values))
    i, j = torch.arange(before, length, device=DEV)[:, None], torch.arange(length, device=DEV)[None, :]
    seen = (j <= i) & ((i - j < window) if window else True)
    scores = torch.einsum("thd,jhd->htj", q.double(), k) * head_dim ** -0.5
    expected = torch.einsum("htj,jhd->thd", torch.softmax(scores.masked_fill(~seen, -math.inf), dim=-1), v)
    # every row written, and within the bound derived above
    assert float((out.view(tokens, q_heads, head_dim).double() - expected).abs().max()) <= 3e-5


def test_32_bit_attention_reports_a_missing_page(ops):
    cache, table, keys, values = paged_setup(torch.float32, [40], 1, 32, 8)
    q = rand(40, 2, 32)
    table[0, 1] = -1
    start, context = torch.tensor([0, 40], dtype=torch.int32, device=DEV), torch.tensor([40], dtype=torch.int32, device=DEV)
    for call in (lambda: ops.attention_f32_prefill(q, cache, table, start, context, 40, None, 1.0),
                 lambda: ops.attention_f32_decode(q[:1], cache, table, context, 40, None, 1.0)):
        call()
        with pytest.raises(ops.KernelError, match="no page"):
            ops.check_device_errors(torch.device(DEV))


@pytest.mark.parametrize("tokens", [1, 3, 16, 17, 64])
@pytest.mark.parametrize("experts,unit,behind,width", [(16, 2, 296, 520), (3, 1, 0, 64), (40, 1, 64, 1000)])
@pytest.mark.parametrize("tiled", [False, True])
def test_products_with_the_chosen_experts_alone(ops, tokens, experts, unit, behind, width, tiled):
    """Both forms against 64-bit arithmetic of the matrices that some token uses: no expert, one, a few, all of them."""
    weight = rand(experts * unit * 128 + behind, width, dtype=torch.bfloat16)
    wide = rand(width, experts * unit * 64 + behind, dtype=torch.bfloat16, seed=1)
    x = rand(tokens, width, dtype=torch.bfloat16, seed=2)
    as_given = ops.tile_weight if tiled else (lambda w: w)
    for used in ([], [experts - 1], [0, experts // 2], list(range(experts))):
        gates = torch.zeros(tokens, experts + 3, device=DEV)
        gates[:, experts:] = 1.0  # columns beyond the experts' say nothing about them
        for i, e in enumerate(used):
            gates[i % tokens, e] = -0.25 if i else 1e-30
        rows = torch.tensor([e in used for e in range(experts)], device=DEV).repeat_interleave(unit * 128)
        rows = torch.cat([rows, torch.ones(behind, dtype=torch.bool, device=DEV)])
        want = x.double() @ weight.double().T
        for expected in (1, len(used) * unit + 3, 10 ** 6):
            got = ops.linear_chosen(x, as_given(weight), gates, experts, unit, False, expected, torch.float32)
            # 32-bit sums of `width` products of about 1 each: the usual bound, width * 2^-24 * sum |x w|, with its random walk
            assert torch.allclose(got[:, rows].double(), want[:, rows], rtol=0, atol=width * 2.0 ** -20), (used, expected)
        hidden = rand(tokens, wide.shape[1], dtype=torch.bfloat16, seed=3)
        columns = torch.tensor([e in used for e in range(experts)], device=DEV).repeat_interleave(unit * 64)
        columns = torch.cat([columns, torch.ones(behind, dtype=torch.bool, device=DEV)])
        want = (hidden * columns).double() @ wide.double().T
        hidden[:, ~columns] = float("nan")  # left out, not multiplied by zero
        got = ops.linear_chosen(hidden, as_given(wide), gates, experts, unit, True, out_dtype=torch.float32)
        assert torch.allclose(got.double(), want, rtol=0, atol=wide.shape[1] * 2.0 ** -20), used
    ops.check_device_errors(torch.device(DEV))


@pytest.mark.parametrize("heads_on", [False, True])
@pytest.mark.parametrize("tokens", [1, 5, 16, 33, 64])
def test_experts_are_the_same_whole_and_chosen(ops, monkeypatch, tokens, heads_on):
    """The part with each product whole and each reading the chosen experts alone, with a shared branch stacked behind the
    experts and without: the gates' zeros stand for what is not read, whatever memory held there."""
    from part_helpers import load_part
    from kirai_b200.parts.experts import RoutedExperts
    from kirai_b200.parts.swiglu import SwiGLU

    shared = SwiGLU("shared.", 256, 192) if heads_on else None
    more = dict(scoring="softmax_corrected", weight_scale=1.0, shared=shared, shared_gate="sg") if heads_on else {}
    part = RoutedExperts("m.", 256, 128, 12, 2, activation="silu_gated", **more)
    load_part(part, torch.bfloat16, seed=3)
    x = rand(tokens, 256, dtype=torch.bfloat16, seed=4)
    results = []
    for up, down in ((False, False), (True, False), (False, True), (True, True)):
        monkeypatch.setattr(ops, "linear_chosen_pays", lambda *a, **k: down if a[6] else up)
        torch.full((tokens, part.up.out_features), float("nan"), dtype=torch.bfloat16, device=DEV)  # what an unwritten column may hold
        results.append(part.forward(x).float())
    ops.check_device_errors(torch.device(DEV))
    for result in results[1:]:
        # the same products in 32-bit sums of another order, then one rounding to bfloat16
        assert float((result - results[0]).abs().max()) <= 2.0 ** -7 * float(results[0].abs().max())


@pytest.mark.parametrize("likely", [1, 2, 33, 511, 512, 513, 3000])
@pytest.mark.parametrize("vocab", [32000, 151936])
def test_sampling_where_few_entries_hold_the_nucleus(ops, likely, vocab):
    """``likely`` entries far above the rest: up to 512 of them are collected and ordered, more are searched for.  Some tie."""
    generator = torch.Generator().manual_seed(likely)
    draws = torch.tensor([0.0, 0.2, 0.5, 0.77, 0.999])
    logits = torch.randn(len(draws), vocab, generator=generator) - 30.0
    for row in logits:
        row[torch.randperm(vocab, generator=generator)[:likely]] = torch.randint(0, 8, (likely,), generator=generator) / 8.0 + 1.0
    for top_p in (0.9, 1.0, 1e-6):
        for temperature in (0.7, 1.0):
            column = lambda v: torch.full((len(draws),), v, device=DEV)  # noqa: E731
            got = ops.sample_rows(logits.to(DEV), column(temperature), column(top_p), draws.to(DEV)).tolist()
            for row, draw in enumerate(draws.tolist()):
                probs = torch.softmax(logits[row].double() / temperature, 0)
                order = torch.argsort(-probs, stable=True)
                running = torch.cumsum(probs[order], 0)
                last = vocab - 1 if top_p >= 1.0 else int(torch.searchsorted(running, torch.tensor(top_p, dtype=torch.float64)))
                place = int((order == got[row]).nonzero())
                # 32-bit sums of up to 3,000 (and 152,000 tiny) terms, formed in another order: 2^-24 a rounding
                slack, threshold = 3e-5, draw * float(running[last])
                before = float(running[place - 1]) if place else 0.0
                assert before - slack <= threshold <= float(running[place]) + slack, (row, top_p, place)
                assert before <= float(running[last]) + slack
    ops.check_device_errors(torch.device(DEV))


@pytest.mark.parametrize("q_heads,kv_heads,head_dim,page_size,form",
                         [(32, 8, 128, 16, {}), (4, 4, 64, 8, {"window": 20}), (8, 1, 96, 64, {"softcap": 5.0}), (6, 2, 48, 1, {"sinks": True}),
                          (4, 2, 128, 16, {"chunk": 48}), (7, 1, 128, 32, {"window": 37, "keep_first": 5})])
def test_decode_attention_of_crowds(ops, q_heads, kv_heads, head_dim, page_size, form):
    """The decode attention for many requests (the longest first) against the plain kernel, with both sizes of CTAs, whole and in
    ranges (more ranges than a request has tiles, too); requests of one token, of whole tiles, of a tile and one, and of equal length."""
    lengths = [1, 150, 16, 17, 300, 5, 64, 33, 64, 150, 1]
    cache, table, keys, values = paged_setup(torch.bfloat16, lengths, kv_heads, head_dim, page_size, seed=5)
    for r, n in enumerate(lengths):
        ops.kv_write(keys[r].to(DEV).contiguous(), values[r].to(DEV).contiguous(), cache, table,
                     torch.full((n,), r, dtype=torch.int32, device=DEV), torch.arange(n, dtype=torch.int32, device=DEV))
    q = rand(len(lengths), q_heads, head_dim, dtype=torch.bfloat16, scale=2.0)
    scale, context = head_dim ** -0.5, torch.tensor(lengths, dtype=torch.int32, device=DEV)
    sinks = rand(q_heads) if form.get("sinks") else None
    options = dict(chunk=form.get("chunk"), softcap=form.get("softcap"), keep_first=form.get("keep_first", 0), sinks=sinks)
    window = form.get("window")
    plain = ops.paged_attention_plain(q.float(), cache.float(), table, torch.arange(len(lengths), dtype=torch.int32, device=DEV), context - 1,
                                      window, scale, **options)
    for warps in (4, 8):
        for splits in (1, 2, 3, 21):
            got = ops.attention_decode_crowd(q, cache, table, context, window, scale, splits, warps, **options)
            # weights and result are rounded to bfloat16 (2^-9 each) on values of up to about 4
            assert float((got.float() - plain).abs().max()) <= 2.5e-2, (warps, splits)
    ops.check_device_errors(torch.device(DEV))


@pytest.mark.parametrize("requests,kv_heads,head_dim", [(511, 1, 64), (512, 2, 128), (203, 4, 128)])
def test_decode_attention_of_the_largest_crowds(ops, requests, kv_heads, head_dim):
    """As many requests as a launch orders by length, and numbers that are no multiple of four; many of equal length.  Every request
    has to be attended once, whatever the place of its length in shared memory."""
    generator = torch.Generator().manual_seed(requests)
    lengths = torch.randint(1, 80, (requests,), generator=generator).tolist()
    cache, table, keys, values = paged_setup(torch.bfloat16, lengths, kv_heads, head_dim, 16, seed=6)
    for r, n in enumerate(lengths):
        ops.kv_write(keys[r].to(DEV).contiguous(), values[r].to(DEV).contiguous(), cache, table,
                     torch.full((n,), r, dtype=torch.int32, device=DEV), torch.arange(n, dtype=torch.int32, device=DEV))
    q = rand(requests, 2 * kv_heads, head_dim, dtype=torch.bfloat16, scale=2.0)
    scale, context = head_dim ** -0.5, torch.tensor(lengths, dtype=torch.int32, device=DEV)
    plain = ops.paged_attention_plain(q.float(), cache.float(), table, torch.arange(requests, dtype=torch.int32, device=DEV), context - 1,
                                      None, scale)
    for warps, splits in ((4, 1), (8, 1), (4, 2)):
        for _ in range(3):
            got = ops.attention_decode_crowd(q, cache, table, context, None, scale, splits, warps)
            # weights and result are rounded to bfloat16 (2^-9 each) on values of up to about 4
            assert float((got.float() - plain).abs().max()) <= 2.5e-2, (warps, splits)
    ops.check_device_errors(torch.device(DEV))


@pytest.mark.parametrize("tokens,rot_dims,norm", [(1, 64, False), (3, 128, True), (255, 64, True), (256, 64, True), (300, 32, False)])
def test_rotated_heads_spread_over_blocks(ops, tokens, rot_dims, norm):
    """Below 256 tokens a token's heads go over several blocks (29 here: a last block with part of its warps idle); every row is
    what the token makes alone, and the rotation's formula."""
    nq, nkv, dim, page = 17, 6, 128, 16
    rows = rand(tokens, (nq + 2 * nkv) * dim, seed=tokens)
    freq = (10000.0 ** (-torch.arange(rot_dims // 2, dtype=torch.float64) * 2 / rot_dims)).float().to(DEV)
    weights = dict(q_norm=(1.0 + 0.1 * rand(dim, seed=1)).contiguous(), k_norm=(1.0 + 0.1 * rand(dim, seed=2)).contiguous(), norm_eps=1e-6) if norm else {}
    pages = -(-tokens // page)
    table = torch.randperm(pages, generator=torch.Generator().manual_seed(3)).int().view(1, -1).to(DEV)
    positions, request = torch.arange(tokens, dtype=torch.int32, device=DEV), torch.zeros(tokens, dtype=torch.int32, device=DEV)

    def prepare(cache, first, last):
        return ops.qkv_rope_write(rows[first:last], nq, nkv, dim, dim, dim, None, None, None, None, freq, 0, rot_dims, cache, table,
                                  request[first:last], positions[first:last], torch.float32, **weights)

    whole, one = (torch.zeros(pages, 2, nkv, page, dim, device=DEV) for _ in range(2))
    q = prepare(whole, 0, tokens)
    alone = torch.cat([prepare(one, t, t + 1) for t in range(tokens)])
    ops.check_device_errors(torch.device(DEV))
    assert torch.equal(q, alone) and torch.equal(whole, one)
    x = rows[:, : nq * dim].double().view(tokens, nq, dim)
    if norm:
        x = x * torch.rsqrt((x * x).mean(-1, keepdim=True) + 1e-6) * weights["q_norm"].double()
    angle = (positions.float()[:, None] * freq[None]).double()
    half = rot_dims // 2
    c, s, a, b = angle.cos()[:, None], angle.sin()[:, None], x[..., :half], x[..., half:rot_dims]
    expected = torch.cat([a * c - b * s, b * c + a * s, x[..., rot_dims:]], dim=-1)
    # a handful of 32-bit operations on values of a few units (the sum of squares has 128 terms in a tree of depth 9)
    assert float((q.double() - expected).abs().max()) <= 16 * 2.0 ** -24 * float(expected.abs().max())


def test_the_error_word_leaves_a_step_beside_its_tokens(ops):
    sampled = torch.tensor([5, 9, 2], dtype=torch.int32, device=DEV)
    results = torch.full((4,), 77, dtype=torch.int32, device=DEV)
    positions, lengths = torch.tensor([3, 4, 5], dtype=torch.int32, device=DEV), torch.tensor([4, 5, 6], dtype=torch.int32, device=DEV)
    flag = ops.error_flag(torch.device(DEV))
    for word in (0, 3):
        flag.fill_(word)
        ops.decode_advance(results[:3], sampled, positions, lengths, results[3:])
        assert results.tolist() == [5, 9, 2, word]
    flag.zero_()
    ops.decode_advance(results[:3], sampled, positions, lengths)
    assert results.tolist() == [5, 9, 2, 3] and positions.tolist() == [6, 7, 8] and lengths.tolist() == [7, 8, 9]


@pytest.mark.parametrize("width", [256, 2048, 2052, 4096, 4100, 8192])
@pytest.mark.parametrize("rows", [148, 149, 740, 741])
def test_row_kernels_on_both_sides_of_where_they_read_early(ops, rows, width):
    """Up to 148 rows, and up to 740 of at most 4,096 columns, a block asks for the whole row at once, then for its parts in turn: the
    same arithmetic, so the same bits as the first rows give alone, and the formulas."""
    stream, y, other = (rand(rows, width, seed=i) for i in (1, 2, 3))
    w, w2 = rand(width, seed=4), rand(width, seed=5)
    gates = torch.rand(rows, 3, generator=torch.Generator().manual_seed(6)).to(DEV)
    unit = lambda x, eps: x.double() / torch.sqrt((x.double() ** 2).mean(-1, keepdim=True) + eps)  # noqa: E731

    def added(n):
        resid = stream[:n].clone()
        copy = ops.norm_add(resid, y[:n].contiguous(), w, 1e-6, torch.bfloat16)
        return resid, copy

    def terms(n):
        resid = stream[:n].clone()
        slots = torch.arange(2 * n, dtype=torch.int32, device=DEV).view(n, 2)
        sorted_rows = torch.cat([y[:n, None], other[:n, None]], dim=1).reshape(2 * n, width).bfloat16()
        copy = ops.terms_norm_add(resid, y[:n].contiguous(), (sorted_rows, slots, gates[:n, 1:].contiguous()), other[:n].contiguous(), gates[:n].contiguous(), 0, (1, 1),
                                  w, 1e-6, torch.bfloat16)
        return resid, copy

    def mean(n):
        return (ops.rms_pair_mean(y[:n].contiguous(), other[:n].contiguous(), w, w2, 1e-6),)

    for run in (added, terms, mean):
        for whole, few in zip(run(rows), run(5)):
            assert torch.equal(whole[:5], few)
    sums = y.double() + gates[:, :1].double() * other.double() + gates[:, 1:2].double() * stream.double()
    sums += gates[:, 1:2].double() * y.bfloat16().double() + gates[:, 2:].double() * other.bfloat16().double()
    # a dozen 32-bit operations on values of up to about 30, and sums of up to 8,192 squares in a tree
    for got, want in ((added(rows)[0], stream.double() + unit(y, 1e-6) * w.double()), (terms(rows)[0], stream.double() + unit(sums, 1e-6) * w.double()),
                      (mean(rows)[0], 0.5 * (unit(y, 1e-6) * w.double() + unit(other, 1e-6) * w2.double()))):
        assert float((got.double() - want).abs().max()) <= 32 * 16.0 * 2.0 ** -24
