"""The float32 engine's own kernels: products on the tensor cores with every operand split into three bfloat16 numbers,
and paged attention of prompt portions and of single tokens, each against 64-bit results at the edges of its tiles."""
import pytest
import torch

from test_gpu_kernels import DEV, K, paged_case  # noqa: F401  (K is a fixture)

pytestmark = pytest.mark.gpu


def operands(M, N, Kd, seed=1, mean=0.0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    a = torch.randn(M, Kd, generator=g, device=DEV) + mean
    w = torch.randn(N, Kd, generator=g, device=DEV) * 0.1 + mean
    return a, w


@pytest.mark.parametrize("M,N,Kd", [(1, 1, 4), (1, 130, 36), (16, 127, 32), (17, 129, 100), (32, 513, 1600), (33, 128, 64), (64, 300, 260),
                                    (65, 1600, 1600), (128, 128, 6400), (129, 257, 96), (300, 1281, 1280), (7, 1600, 6400)])
def test_split_product(K, M, N, Kd):
    """Against 64 bits: within the bound of float32 summation of the terms' sizes (one rounding a k block of 32 and its
    few cut-off additions), and over all outputs no further off than one chain of float32 multiply-adds an output."""
    for mean in (0.0, 1.0):
        a, w = operands(M, N, Kd, mean=mean)
        want, size = a.double() @ w.double().t(), a.double().abs() @ w.double().abs().t()
        got = K.gemm_split(a, w)
        # a k block: 12 additions into the accumulator, each cut off at 2^-23 of what has been added so far; the blocks'
        # sums, and the blocks of a cluster, one rounding each; the three products left out, 3 x 2^-25 of their term
        allowed = size * (14 * 2.0 ** -23 + (Kd / 32 + 9) * 2.0 ** -24)
        assert ((got.double() - want).abs() <= allowed).all()
        plain = K.gemm_simt(a, w)
        # (with a handful of outputs either of the two may be the lucky one)
        if M * N >= 1024:
            assert (got.double() - want).norm() <= (plain.double() - want).norm()
        assert torch.equal(got, K.gemm_split(a, w)), "two runs are bit-equal"
    bias, stream = torch.randn(N, device=DEV), torch.randn(M, N, device=DEV)
    u = want + bias.double()
    full = K.gemm_split(a, w, bias, residual=stream.clone(), activation="gelu")
    exact = 0.5 * u * (1 + torch.erf(u / 2 ** 0.5)) + stream.double()
    assert ((full.double() - exact).abs() <= 2 * allowed + 1e-6 * (1 + u.abs())).all()
    in_place = stream.clone()
    assert K.gemm_split(a, w, bias, residual=in_place, out=in_place).data_ptr() == in_place.data_ptr()
    assert ((in_place.double() - u - stream.double()).abs() <= allowed + 1e-6 * (1 + u.abs())).all()
    assert K.read_error_flag(DEV) == 0


@pytest.mark.parametrize("tile,M", [(16, 9), (32, 50), (64, 130), (128, 131)])
def test_split_product_in_any_tile_and_cluster(K, tile, M):
    N, Kd = 390, 416
    a, w = operands(M, N, Kd, seed=3)
    wide = torch.full((M, N + 8), 7.0, device=DEV)
    want = a.double() @ w.double().t()
    for splits in (1, 2, 3, 8):
        got = K.gemm_split(a, w, out=wide[:, 4:4 + N], token_tile=tile, splits=splits)
        assert (got.double() - want).abs().max() < 2e-5
        assert bool((wide[:, :4] == 7).all()) and bool((wide[:, 4 + N:] == 7).all())
    # operands inside wider rows
    big_a, big_w = torch.randn(M, Kd + 12, device=DEV), torch.randn(N, Kd + 4, device=DEV)
    got = K.gemm_split(big_a[:, 4:4 + Kd], big_w[:, 4:4 + Kd], token_tile=tile)
    assert (got.double() - big_a[:, 4:4 + Kd].double() @ big_w[:, 4:4 + Kd].double().t()).abs().max() < 4e-4
    assert K.read_error_flag(DEV) == 0


@pytest.mark.parametrize("M", [5, 40, 70, 200])
def test_split_product_of_values_that_have_no_three_parts(K, M):
    """Infinities, NaN, numbers that bfloat16 rounds to infinity, sums that overflow: what the float32 kernel gives."""
    a, w = operands(M, 200, 160, seed=5)
    a[1, 7], a[2, 9], a[3, 30], a[4, 31] = float("inf"), float("nan"), 3.4e38, -float("inf")
    w[5, 11], w[6, 12], w[130, 40] = float("inf"), -3.395e38, float("nan")
    a[0, :40] = 1e30
    w[8, :40] = 1e12
    w[9, :40] = 1e-30
    got, plain = K.gemm_split(a, w), K.gemm_simt(a, w)
    finite = torch.isfinite(plain)
    assert torch.equal(torch.isnan(plain), torch.isnan(got)) and torch.equal(finite, torch.isfinite(got))
    odd = ~finite & ~torch.isnan(plain)
    assert torch.equal(got[odd], plain[odd]) and bool(odd.any())
    assert ((got - plain)[finite].abs() <= 1e-4 * (1 + plain[finite].abs())).all()
    tiny = torch.full((M, 160), 1e-20, device=DEV)
    assert torch.allclose(K.gemm_split(tiny, w[20:60]) * 1e20, w[20:60].sum(1).expand(M, -1), atol=2e-5)


def test_a_row_beside_others(K):
    """What a row's bits depend on. In the split product K is cut among the blocks of a cluster by the number of tiles, so a row
    has the same bits among 1 to 128 rows here, where eight blocks share a tile, and others among more, within the error of the
    sums' order; the product on the CUDA cores gives a row the same bits whatever is beside it."""
    a, w = operands(300, 1600, 1600, seed=7)
    size = a[:1].double().abs() @ w.double().abs().t()
    alone, plain = K.gemm_split(a[:1], w), K.gemm_simt(a[:1], w)
    for M in (2, 16, 17, 33, 128, 129, 300):
        got = K.gemm_split(a[:M], w)[:1]
        assert K._split_plan(M, 1600, 1600, 148)[0] == (8 if M <= 128 else 5 if M <= 256 else 3)
        assert torch.equal(got, alone) == (M <= 128)
        # every order rounds the sums of 50 k blocks and of the cluster's blocks, at most once each
        assert ((got.double() - alone.double()).abs() <= 2 * (50 + 8) * 2.0 ** -24 * size).all()
        assert torch.equal(K.gemm_simt(a[:M], w)[:1], plain)


def test_which_float32_products_are_split(K):
    from types import SimpleNamespace
    from damendaemon_b200.parts.linear import linear, splits_float32
    assert splits_float32(1600, 1600) and splits_float32(1024, 1024) and not splits_float32(512, 512)
    a, w = operands(8, 1600, 1600)
    auto, plain = SimpleNamespace(gemm="auto"), SimpleNamespace(gemm="simt")
    assert torch.equal(linear(auto, a, w), K.gemm_split(a, w)) and torch.equal(linear(plain, a, w), K.gemm_simt(a, w))
    # rows that start off a 16-byte boundary stay on the CUDA cores
    shifted = torch.randn(8, 1601, device=DEV)[:, 1:]
    assert torch.equal(linear(auto, shifted, w), K.gemm_simt(shifted, w))
    # ... and so do rows that lie over one another, which no tensor map describes
    for rows in (a[:1].expand(8, 1600), torch.randn(8 * 1600, device=DEV).as_strided((8, 1600), (16, 1))):
        assert not K.gemm_split_fits(rows, w) and torch.equal(linear(auto, rows, w), K.gemm_simt(rows.contiguous(), w))
    with pytest.raises(K.KernelError, match="over one another"):
        K.gemm_split(a[:1].expand(8, 1600), w)
    one = a.as_strided((1, 1600), (0, 1))
    assert torch.equal(linear(auto, one, w), K.gemm_split(a[:1], w))


@pytest.mark.parametrize("M,N,Kd", [(1, 1, 4), (8, 7, 132), (3, 1000, 1600), (8, 9000, 256), (5, 6400, 1792), (8, 1600, 1796), (2, 1600, 6400),
                                    (8, 3001, 14336)])
def test_streamed_product(K, M, N, Kd):
    """Up to eight rows through the CUDA cores: the last group of rows smaller, several groups a warp, K that ends inside a box,
    one to eight blocks on a sum. Within the bound of chains of K / 64 float32 multiply-adds and, over all outputs, no further
    from 64 bits than the split product, which serves more rows."""
    for mean in (0.0, 1.0):
        a, w = operands(M, N, Kd, mean=mean)
        want, size = a.double() @ w.double().t(), a.double().abs() @ w.double().abs().t()
        got = K.gemm_stream(a, w)
        # a lane's pair of sums takes at most two products a sub-box of 128 k; the rest is float64 and one last rounding
        assert ((got.double() - want).abs() <= size * (2 * (Kd / 128 + 1) + 1) * 2.0 ** -24).all()
        if M * N >= 1024 and mean == 0.0:
            assert (got.double() - want).norm() <= (K.gemm_split(a, w).double() - want).norm()
        assert torch.equal(got, K.gemm_stream(a, w)), "two runs are bit-equal"
        assert torch.equal(got[:1], K.gemm_stream(a[:1], w)), "a row does not depend on the others"
    bias, stream = torch.randn(N, device=DEV), torch.randn(M, N, device=DEV)
    u, allowed = want + bias.double(), size * (2 * (Kd / 128 + 1) + 1) * 2.0 ** -24
    wide = torch.full((M, N + 8), 7.0, device=DEV)
    full = K.gemm_stream(a, w, bias, residual=stream, activation="gelu", out=wide[:, 4:4 + N])
    exact = 0.5 * u * (1 + torch.erf(u / 2 ** 0.5)) + stream.double()
    assert ((full.double() - exact).abs() <= 2 * allowed + 1e-6 * (1 + u.abs())).all()
    assert bool((wide[:, :4] == 7).all()) and bool((wide[:, 4 + N:] == 7).all())
    in_place = stream.clone()
    assert K.gemm_stream(a, w, bias, residual=in_place, out=in_place).data_ptr() == in_place.data_ptr()
    assert ((in_place.double() - u - stream.double()).abs() <= allowed + 1e-6 * (1 + u.abs())).all()
    # operands inside wider rows, whose neighbours are no numbers
    big_a, big_w = torch.full((M, Kd + 8), float("nan"), device=DEV), torch.full((N, Kd + 8), float("nan"), device=DEV)
    big_a[:, 4:4 + Kd], big_w[:, 4:4 + Kd] = a, w
    assert torch.equal(K.gemm_stream(big_a[:, 4:4 + Kd], big_w[:, 4:4 + Kd]), got)
    assert K.read_error_flag(DEV) == 0


def test_streamed_product_of_values_that_are_not_finite(K):
    a, w = operands(5, 200, 160, seed=5)
    a[1, 7], a[2, 9], a[3, 30], a[4, 31] = float("inf"), float("nan"), 3.4e38, -float("inf")
    w[5, 11], w[6, 12], w[130, 40] = float("inf"), -3.395e38, float("nan")
    got, plain = K.gemm_stream(a, w), K.gemm_simt(a, w)
    finite = torch.isfinite(plain)
    assert torch.equal(torch.isnan(plain), torch.isnan(got)) and torch.equal(finite, torch.isfinite(got))
    assert ((got - plain)[finite].abs() <= 1e-4 * (1 + plain[finite].abs())).all()


def test_which_float32_products_are_streamed(K):
    from types import SimpleNamespace
    from damendaemon_b200.parts.linear import linear, streams_float32
    assert streams_float32(8, 3072, 1024) and not streams_float32(9, 3072, 1024) and \
        not streams_float32(1, 1600, 1600) and not streams_float32(8, 50257, 1600)
    auto, plain = SimpleNamespace(gemm="auto"), SimpleNamespace(gemm="simt")
    a, w = operands(9, 3072, 1024)
    assert torch.equal(linear(auto, a[:8], w), K.gemm_stream(a[:8], w)) and torch.equal(linear(auto, a, w), K.gemm_split(a, w))
    assert torch.equal(linear(plain, a[:8], w), K.gemm_simt(a[:8], w))
    one = a.as_strided((1, 1024), (0, 1))
    assert torch.equal(linear(auto, one, w), K.gemm_stream(a[:1], w))
    for rows in (a[:1].expand(8, 1024), torch.randn(8, 1025, device=DEV)[:, 1:]):
        assert torch.equal(linear(auto, rows, w), K.gemm_simt(rows.contiguous() if rows.stride(0) == 0 else rows, w))
    with pytest.raises(K.KernelError, match="takes up to 8 rows"):
        K.gemm_stream(a, w)
    with pytest.raises(K.KernelError, match="over one another"):
        K.gemm_stream(a[:1].expand(8, 1024), w)


@pytest.mark.parametrize("N,Kd,streamed", [
    # measured at 1 and 8 rows, split product / stream (us)
    (4096, 4096, False),        # 18.0 / 26.6: more rows than the clusters that are resident take in one round
    (65536, 128, False),        # 14.3 / 24.4: little to sum for every row
    (11008, 4096, False), (4096, 11008, False), (5632, 2048, False), (50000, 1000, False), (32000, 1536, False), (3200, 6400, False),
    (2048, 2048, True),         # 15.2 / 8.1: more clusters of the split product than are resident
    (1600, 6400, True), (1280, 5120, True), (1024, 4096, True), (25600, 1600, True), (512, 8192, True), (4800, 1600, True)])
def test_a_matrix_is_streamed_where_that_is_ahead(K, N, Kd, streamed):
    from types import SimpleNamespace
    from damendaemon_b200.parts.linear import linear, streams_float32
    assert streams_float32(1, N, Kd) == streamed and streams_float32(8, N, Kd) == streamed and not streams_float32(9, N, Kd)
    a, w = operands(3, N, Kd)
    assert torch.equal(linear(SimpleNamespace(gemm="auto"), a, w), (K.gemm_stream if streamed else K.gemm_split)(a, w))


def test_resident_clusters_of_the_streamed_product(K):
    """Asked first for a part of the GPU and by several threads: the answer for all of it is not that of the part."""
    from concurrent.futures import ThreadPoolExecutor
    ask = K.library("core").dd_gemm_stream_clusters
    assert ask(2, 16) <= 8 and ask(0, 148) == 0 and ask(9, 148) == 0 and ask(8, 7) == 0
    with ThreadPoolExecutor(8) as pool:
        for n, got in enumerate(pool.map(lambda n: [ask(n, 148) for _ in range(50)], range(1, 9)), start=1):
            assert len(set(got)) == 1 and 148 // n // 2 < got[0] <= 148 // n


def run_of_entries(dtype, entries, keys, heads, kv_heads, d, page=16, seed=11):
    """Queries of `entries` requests with `keys` tokens each, their caches and block tables: q [entries * keys, ...] is what a
    prompt of whole requests brings, its last row of every entry what a decode step brings."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    blocks = -(-keys // page)
    q = torch.randn(entries * keys, heads * d, generator=g, device=DEV).to(dtype)
    k, v = (torch.randn(entries, keys, kv_heads, d, generator=g, device=DEV).to(dtype) for _ in range(2))
    table = torch.randperm(entries * blocks, generator=g, device=DEV).to(torch.int32).view(entries, blocks)

    def cache(k, v):
        pages = torch.zeros(entries * blocks, 2, kv_heads, page, d, dtype=dtype, device=DEV)
        for side, x in enumerate((k, v)):
            padded = torch.nn.functional.pad(x, (0, 0, 0, 0, 0, blocks * page - keys)).view(entries, blocks, page, kv_heads, d)
            pages[table.long(), side] = padded.transpose(2, 3)
        return pages
    return q, k, v, table, cache


SIZES = [(3, 3, 16, 16), (4, 2, 48, 8), (5, 5, 64, 16), (6, 2, 32, 12), (2, 1, 128, 32), (2, 2, 20, 4), (3, 1, 100, 16)]


@pytest.mark.parametrize("heads,kv_heads,d,page", SIZES)
@pytest.mark.parametrize("window", [None, 70])
def test_prompt_attention(K, heads, kv_heads, d, page, window):
    lengths, new = [64, 1, 65, 200, 331], [64, 1, 1, 129, 64]
    c = paged_case(K, torch.float32, heads, kv_heads, d, page, lengths, new, window, 1)
    assert K.attention_cores_supported(c["q"], c["cache"])
    start = torch.tensor([0] + torch.tensor(new).cumsum(0).tolist(), dtype=torch.int32, device=DEV)
    pos0 = torch.tensor([n - m for n, m in zip(lengths, new)], dtype=torch.int32, device=DEV)
    for splits in (1, 2, 3, 4):
        got = K.attention_f32_prompt(c["q"], c["cache"], start, pos0, c["table"], heads, c["scale"], window, n_splits=splits)
        assert (got.cpu().double() - c["ref"]).abs().max() < 2e-5
    # the chunked mask and the gate, as the general kernel has them
    gate = torch.randn(sum(new), heads, device=DEV)
    more = dict(chunk=40, gate=gate)
    want = K.attention_rows(c["q"], c["cache"], c["ent"], c["pos"], c["table"], heads, c["scale"], window, **more)
    got = K.attention_f32_prompt(c["q"], c["cache"], start, pos0, c["table"], heads, c["scale"], window, n_splits=2, **more)
    assert (got - want).abs().max() < 2e-5 and K.read_error_flag(DEV) == 0


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("heads,kv_heads,d,page", SIZES)
@pytest.mark.parametrize("splits", [1, 3, 8])
def test_single_token_attention(K, heads, kv_heads, d, page, splits, dtype):
    if d * dtype.itemsize % 16:
        pytest.skip("rows that are not whole 16-byte pieces")
    lengths = [1, 2, 63, 64, 65, 300, 517]
    for window, chunk in ((None, None), (70, None), (None, 40)):
        c = paged_case(K, dtype, heads, kv_heads, d, page, lengths, [1] * len(lengths), window, 1, store=False)
        assert K.attention_cores_supported(c["q"], c["cache"])
        k = c["packed"][:, heads * d:(heads + kv_heads) * d]
        v = c["packed"][:, (heads + kv_heads) * d:]
        stored = c["cache"].clone()
        K.kv_store(k, v, c["ent"], c["pos"], c["table"], stored)
        gate = torch.randn(len(lengths), heads, device=DEV).to(dtype) if chunk else None
        got = K.attention_tokens(c["q"], c["cache"], c["pos"], c["table"], heads, c["scale"], window, n_splits=splits, k_new=k, v_new=v,
                                 chunk=chunk, gate=gate)
        assert torch.equal(torch.nan_to_num(c["cache"], nan=5.0), torch.nan_to_num(stored, nan=5.0)), "the new keys and values are in the cache"
        # weights and sums are float32 whatever the storage type: a bfloat16 result is off by its own rounding, half of its
        # spacing, which is 2^-7 of a power of two: at most 2^-8 of the value (beside the general kernel's, which is rounded as
        # well, twice that)
        rounding = 0.0 if dtype == torch.float32 else 2.0 ** -8
        if chunk is None:
            assert ((got.cpu().double() - c["ref"]).abs() <= rounding * c["ref"].abs() + 2e-5).all()
        want = K.attention_rows(c["q"], stored, c["ent"], c["pos"], c["table"], heads, c["scale"], window, chunk=chunk, gate=gate).double()
        assert ((got.double() - want).abs() <= 2 * (1 + 2.0 ** -7) * rounding * want.abs() + 2e-5).all()
        again = K.attention_tokens(c["q"], stored, c["pos"], c["table"], heads, c["scale"], window, n_splits=splits, chunk=chunk, gate=gate)
        assert torch.equal(got, again) and K.read_error_flag(DEV) == 0


def plain_decode(q, k, v, heads, lengths, scale):
    """One query an entry in 64 bits: q [entries, heads * d], k and v [entries, keys, kv_heads, d] with `lengths` keys of each."""
    q, k, v = q.double().view(len(lengths), heads, -1), k.double(), v.double()
    rep = heads // k.shape[2]
    s = torch.einsum("ehd,ekhd->ehk", q, k.repeat_interleave(rep, 2)) * scale
    s = s.masked_fill(torch.arange(k.shape[1], device=DEV)[None, None] >= torch.tensor(lengths, device=DEV)[:, None, None], float("-inf"))
    return torch.einsum("ehk,ekhd->ehd", torch.softmax(s, -1), v.repeat_interleave(rep, 2)).reshape(len(lengths), -1)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("heads,kv_heads,d,page", [(4, 1, 64, 16), (2, 2, 48, 24), (2, 1, 128, 64)])
def test_single_token_attention_over_long_contexts(K, heads, kv_heads, d, page, dtype):
    """Contexts around and beyond 4,096 keys, where the rule cuts a token's keys into more pieces, pages of a power of two and
    others; in every number of pieces. Weights and sums are float32: a bfloat16 result is off by its own rounding alone."""
    from types import SimpleNamespace
    from damendaemon_b200.parts.paged_attention import token_splits
    lengths = [4095, 4096, 4097, 9001, 17]
    q, k, v, table, cache = run_of_entries(dtype, len(lengths), max(lengths), heads, kv_heads, d, page=page)
    q, cache = q.view(len(lengths), max(lengths), -1)[:, -1].contiguous(), cache(k, v)
    pos = torch.tensor(lengths, dtype=torch.int32, device=DEV) - 1
    want = plain_decode(q, k, v, heads, lengths, d ** -0.5)
    for context, most in ((4096, 4), (4097, 8)):
        assert token_splits(SimpleNamespace(sm_count=148, split_context=context), len(lengths), heads) == most
    for splits in (1, 4, 8):
        got = K.attention_tokens(q, cache, pos, table, heads, d ** -0.5, n_splits=splits)
        allowed = 2e-6 if dtype == torch.float32 else 2.0 ** -8 * want.abs() + 2e-5
        assert ((got.double() - want).abs() <= allowed).all()
    assert K.read_error_flag(DEV) == 0


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_long_contexts_are_not_slower_than_through_the_general_kernel(K, dtype):
    """8 requests x 32 heads of 128 in groups of four at long contexts, which the general kernel read faster while the
    single-token kernel looked its pages up one after the other."""
    heads, kv_heads, d, keys = 32, 8, 128, 4000 if dtype == torch.bfloat16 else 8000
    q, k, v, table, cache = run_of_entries(dtype, 8, keys, heads, kv_heads, d)
    q, cache = q.view(8, keys, -1)[:, -1].contiguous(), cache(k, v)
    pos, ent = torch.full((8,), keys - 1, dtype=torch.int32, device=DEV), torch.arange(8, dtype=torch.int32, device=DEV)

    def fastest(call):
        times = []
        for _ in range(10):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(10):
                call()
            b.record()
            torch.cuda.synchronize()
            times.append(a.elapsed_time(b))
        return min(times)

    tokens = fastest(lambda: K.attention_tokens(q, cache, pos, table, heads, d ** -0.5))
    general = fastest(lambda: K.attention_rows(q, cache, ent, pos, table, heads, d ** -0.5, n_splits=10))
    print(f"{tokens * 100:.1f} us, general kernel {general * 100:.1f} us")
    assert tokens < general


@pytest.mark.parametrize("heads,kv_heads,d,dtype,tokens,kernel", [
    (25, 25, 64, torch.bfloat16, 1, "attention_decode"), (25, 25, 64, torch.bfloat16, 8, "attention_decode"),
    (2, 2, 128, torch.bfloat16, 1, "attention_decode"),
    (10, 2, 64, torch.bfloat16, 8, "attention_tokens"), (3, 3, 16, torch.bfloat16, 5, "attention_tokens"),
    (25, 25, 64, torch.float32, 8, "attention_tokens"), (2, 1, 132, torch.float32, 3, "attention_rows")])
def test_which_kernel_a_decode_step_takes(K, monkeypatch, heads, kv_heads, d, dtype, tokens, kernel):
    """Groups and small heads: the kernel of whole rows; sizes that the tensor-core decode kernels take go to those, however
    few tokens there are. Whichever it is, the result is the general kernel's."""
    from types import SimpleNamespace
    from damendaemon_b200.engine.context import StepContext
    from damendaemon_b200.parts import paged_attention as pa
    lengths = [40 + 7 * i for i in range(tokens)]
    c = paged_case(K, dtype, heads, kv_heads, d, 16, lengths, [1] * tokens, None, 1, store=False)
    q, k, v = c["packed"].split([heads * d, kv_heads * d, kv_heads * d], dim=1)
    ctx = StepContext(tokens, tokens, 0, None, c["pos"], c["ent"], None, None, torch.arange(tokens + 1, dtype=torch.int32, device=DEV), c["pos"],
                      {"all": c["table"]}, decode_only=True, split_context=1024, n_single=tokens,
                      runtime=SimpleNamespace(attention="auto", attention_tuning=pa.AttentionTuning()))
    cache = SimpleNamespace(kv=c["cache"], group=SimpleNamespace(name="all"), writable=True)
    called = []
    for name in ("attention_tokens", "attention_decode", "attention_rows"):
        monkeypatch.setattr(K, name, lambda *a, _f=getattr(K, name), _n=name, **m: (called.append(_n), _f(*a, **m))[1])
    got = pa.paged_attention(ctx, q, k, v, cache, heads, c["scale"])
    assert called == [kernel]
    assert (got.cpu().double() - c["ref"]).abs().max() < (2e-5 if dtype == torch.float32 else 2e-2) and K.read_error_flag(DEV) == 0


@pytest.mark.parametrize("heads,kv_heads,d,tokens,single,most", [(25, 25, 64, 8, 8, 1), (25, 25, 64, 1, 1, 1), (2, 2, 128, 2, 2, 1),
                                                                 (25, 25, 64, 40, 4, 2), (25, 25, 64, 40, 0, 1), (25, 5, 64, 40, 0, 1)])
def test_steps_of_the_tensor_core_sizes_ask_for_no_other_kernel(K, monkeypatch, heads, kv_heads, d, tokens, single, most):
    """An eager step asks these questions for every layer, on the host: what a decode step, a mixed one and a prompt may ask
    about the kernels of sizes that the tensor-core ones refuse is nothing, and about the decode kernels once each."""
    from types import SimpleNamespace
    from damendaemon_b200.engine.context import StepContext
    from damendaemon_b200.parts import paged_attention as pa
    new = [1] * single + ([tokens - single] if tokens > single else [])
    c = paged_case(K, torch.bfloat16, heads, kv_heads, d, 16, [40 + n for n in new], new, None, 1, store=False)
    q, k, v = c["packed"].split([heads * d, kv_heads * d, kv_heads * d], dim=1)
    start = torch.tensor([0] + torch.tensor(new).cumsum(0).tolist(), dtype=torch.int32, device=DEV)
    pos0 = torch.full((len(new),), 40, dtype=torch.int32, device=DEV)
    ctx = StepContext(tokens, len(new), 0, None, c["pos"], c["ent"], None, None, start, pos0, {"all": c["table"]}, decode_only=tokens == single,
                      split_context=1024, n_single=single, runtime=SimpleNamespace(attention="auto", attention_tuning=pa.AttentionTuning()))
    cache = SimpleNamespace(kv=c["cache"], group=SimpleNamespace(name="all"), writable=True)
    asked = []
    for name in ("attention_cores_supported", "attention_decode_supported", "attention_decode_pages_supported"):
        monkeypatch.setattr(K, name, lambda *a, _f=getattr(K, name), _n=name, **m: (asked.append(_n), _f(*a, **m))[1])
    got = pa.paged_attention(ctx, q, k, v, cache, heads, c["scale"])
    assert asked.count("attention_cores_supported") == 0 and len(asked) <= most
    assert (got.cpu().double() - c["ref"]).abs().max() < 2e-2 and K.read_error_flag(DEV) == 0


def test_a_missing_page_is_reported(K):
    lengths = [40, 90]
    c = paged_case(K, torch.float32, 2, 2, 64, 16, lengths, [1, 1], None, 1)
    table = c["table"].clone()
    table[1, 2] = -1
    got = K.attention_tokens(c["q"], c["cache"], c["pos"], table, 2, c["scale"])
    assert K.read_error_flag(DEV) == 4 and torch.isfinite(got).all()
    start, pos0 = (torch.tensor(x, dtype=torch.int32, device=DEV) for x in ([0, 1, 2], [39, 89]))
    got = K.attention_f32_prompt(c["q"], c["cache"], start, pos0, table, 2, c["scale"])
    assert K.read_error_flag(DEV) == 4 and torch.isfinite(got).all()
    table[0, 2] = 1000
    packed = c["packed"]
    K.attention_tokens(c["q"], c["cache"], c["pos"], table, 2, c["scale"], k_new=packed[:, 128:256], v_new=packed[:, 256:])
    assert K.read_error_flag(DEV) & 2


MASKS = [(None, None), (40, None), (None, 48)]


def seen(keys, window, chunk):
    i, j = torch.arange(keys, device=DEV)[:, None], torch.arange(keys, device=DEV)[None, :]
    visible = j <= i
    if window:
        visible &= j > i - window
    if chunk:
        visible &= j // chunk == i // chunk
    return visible


@pytest.mark.parametrize("window,chunk", MASKS)
@pytest.mark.parametrize("heads,kv_heads,d", [(2, 2, 64), (2, 1, 16), (1, 1, 128)])
def test_a_value_that_is_not_finite_reaches_only_queries_that_see_it(K, heads, kv_heads, d, window, chunk):
    """Prompts of 150 tokens, each with one infinite or NaN value row at another place: queries that do not see it have the
    bits of the run without it, queries that do are not finite."""
    keys, places = 150, [0, 1, 30, 63, 64, 65, 100, 127, 128, 148, 149]
    q, k, v, table, cache = run_of_entries(torch.float32, len(places), keys, heads, kv_heads, d)
    start = torch.arange(len(places) + 1, dtype=torch.int32, device=DEV) * keys
    pos0 = torch.zeros(len(places), dtype=torch.int32, device=DEV)
    visible = seen(keys, window, chunk)
    for splits in (1, 3):
        more = dict(n_splits=splits, chunk=chunk)
        clean = K.attention_f32_prompt(q, cache(k, v), start, pos0, table, heads, d ** -0.5, window, **more).view(len(places), keys, -1)
        for value in (float("inf"), -float("inf"), float("nan")):
            spoilt = v.clone()
            for e, j in enumerate(places):
                spoilt[e, j] = value
            got = K.attention_f32_prompt(q, cache(k, spoilt), start, pos0, table, heads, d ** -0.5, window, **more).view(len(places), keys, -1)
            for e, j in enumerate(places):
                sees = visible[:, j]
                assert torch.equal(got[e, ~sees], clean[e, ~sees])
                assert not bool(torch.isfinite(got[e, sees]).any())
    assert K.read_error_flag(DEV) == 0


@pytest.mark.parametrize("window,chunk", MASKS)
@pytest.mark.parametrize("heads,kv_heads,d", [(2, 2, 64), (2, 1, 16), (1, 1, 128)])
def test_a_score_that_is_not_a_number_shows_in_a_prompt(K, heads, kv_heads, d, window, chunk):
    """One NaN key: every query that sees it has no result, the others have theirs; a NaN query alone has none."""
    keys, places = 150, [0, 1, 30, 63, 64, 65, 100, 127, 128, 148, 149]
    q, k, v, table, cache = run_of_entries(torch.float32, len(places), keys, heads, kv_heads, d)
    start = torch.arange(len(places) + 1, dtype=torch.int32, device=DEV) * keys
    pos0 = torch.zeros(len(places), dtype=torch.int32, device=DEV)
    visible, spoilt, odd = seen(keys, window, chunk), k.clone(), q.clone().view(len(places), keys, -1)
    for e, j in enumerate(places):
        spoilt[e, j] = odd[e, j] = float("nan")
    for splits in (1, 2, 4):
        more = dict(n_splits=splits, chunk=chunk)
        clean = K.attention_f32_prompt(q, cache(k, v), start, pos0, table, heads, d ** -0.5, window, **more).view(len(places), keys, -1)
        bad_key = K.attention_f32_prompt(q, cache(spoilt, v), start, pos0, table, heads, d ** -0.5, window, **more).view(len(places), keys, -1)
        bad_query = K.attention_f32_prompt(odd.view(q.shape), cache(k, v), start, pos0, table, heads, d ** -0.5, window, **more).view(len(places), keys, -1)
        for e, j in enumerate(places):
            sees, itself = visible[:, j], torch.arange(keys, device=DEV) == j
            assert torch.equal(bad_key[e, ~sees], clean[e, ~sees]) and bool(torch.isnan(bad_key[e, sees]).all())
            assert torch.equal(bad_query[e, ~itself], clean[e, ~itself]) and bool(torch.isnan(bad_query[e, j]).all())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("heads,kv_heads,d", [(2, 2, 64), (2, 1, 16), (1, 1, 128)])
def test_a_score_that_is_not_a_number_shows_in_a_single_token(K, heads, kv_heads, d, dtype):
    """70 requests of 70 keys, request j with a NaN key at j: no result, wherever the key falls among warps, groups of lanes and
    blocks; in requests of one key as well, and for a NaN query."""
    for keys in (70, 1):
        q, k, v, table, cache = run_of_entries(dtype, 70, keys, heads, kv_heads, d)
        q = q.view(70, keys, -1)[:, -1].contiguous()
        pos = torch.full((70,), keys - 1, dtype=torch.int32, device=DEV)
        bad, odd = k.clone(), q.clone()
        bad[torch.arange(70), torch.arange(70) % keys] = float("nan")
        odd[::2] = float("nan")
        for splits in (1, 2, 3, 8):
            for window in (None, 69):
                clean = K.attention_tokens(q, cache(k, v), pos, table, heads, d ** -0.5, window, n_splits=splits)
                got = K.attention_tokens(q, cache(bad, v), pos, table, heads, d ** -0.5, window, n_splits=splits)
                hidden = window is not None and keys > window                 # then request 0 does not see its NaN key
                assert bool(torch.isnan(got[1 if hidden else 0:]).all()) and (not hidden or torch.equal(got[0], clean[0]))
                got = K.attention_tokens(odd, cache(k, v), pos, table, heads, d ** -0.5, window, n_splits=splits)
                assert bool(torch.isnan(got[::2]).all()) and torch.equal(got[1::2], clean[1::2])
            # the step's own key, which comes from the projection
            packed = torch.cat([q, bad[:, -1].reshape(70, -1), v[:, -1].reshape(70, -1)], dim=1)
            parts = packed.split([heads * d, kv_heads * d, kv_heads * d], dim=1)
            got = K.attention_tokens(parts[0], cache(k, v), pos, table, heads, d ** -0.5, n_splits=splits, k_new=parts[1], v_new=parts[2])
            clean = K.attention_tokens(q, cache(k, v), pos, table, heads, d ** -0.5, n_splits=splits)
            last = torch.arange(70, device=DEV) % keys == keys - 1
            assert bool(torch.isnan(got[last]).all()) and torch.equal(got[~last], clean[~last])
    assert K.read_error_flag(DEV) == 0


def test_admission_counts_the_planes_of_the_split_products(K):
    """What an engine promises to fit before it allocates its cache covers the largest step: 8,192 tokens of prompts through a
    layer whose inner products are split take no more than the estimate; and only products that are split count."""
    from damendaemon_b200.engine import Engine, StepEntry
    from damendaemon_b200.registry import architecture_of
    config = {"architectures": ["GPT2LMHeadModel"], "model_type": "gpt2", "n_layer": 1, "n_embd": 512, "n_head": 8, "n_inner": 2048,
              "vocab_size": 300, "n_positions": 1024}
    arch = architecture_of(config)
    tensors = arch.random_tensors(arch.parse_config(config), 1, torch.float32)
    made = {}
    for dtype, gemm in (("float32", "auto"), ("float32", "simt"), ("bfloat16", "auto")):
        made[dtype, gemm] = Engine(config=config, tensors=tensors, dtype=dtype, gemm=gemm, kv_tokens=8192, max_requests=8)
    engine = made["float32", "auto"]
    planes = K.gemm_split_plane_bytes(8192, 2048, 128)
    assert planes == 8192 * 2048 * 6
    assert engine.workspace_bytes - made["float32", "simt"].workspace_bytes == planes
    assert made["bfloat16", "auto"].workspace_bytes < made["float32", "simt"].workspace_bytes
    entries = [StepEntry(r, [(7 * i + r) % 300 for i in range(1024)], [1023]) for r in range(8)]
    engine.step(entries, end=range(8))                  # (the step's metadata and the error word are allocated)
    torch.cuda.synchronize()
    held = torch.cuda.memory_allocated()
    torch.cuda.reset_peak_memory_stats()
    engine.step(entries, end=range(8))
    assert planes < torch.cuda.max_memory_allocated() - held <= engine.workspace_bytes


def test_plans_that_are_kept_are_bounded(K):
    assert K._split_plan.cache_info().maxsize <= 4096
    for M in (1, 16, 17, 33, 65, 128, 129, 300, 5000):
        splits, tile = K._split_plan(M, 1600, 1600, 148)
        assert tile == (16 if M <= 16 else 32 if M <= 32 else 64 if M <= 64 else 128) and 1 <= splits <= 8
