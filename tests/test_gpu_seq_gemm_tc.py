"""The tensor-core matrix product of steps with more than 16 rows (csrc/seq/seq_gemm_tc.cu) against float64, at the sizes where
its tiles end: rows around 128, columns around 32 / 64 / 128 / 256, k around 64, odd row lengths of C, groups without rows.

Tolerances: operands are bf16 and products exact, so an fp32 result differs from float64 by the rounding of a sum of K terms:
K 2^-24 in the worst case, about sqrt(K) 2^-24 for random signs; 1e-5 covers K <= 1056 with a tensor core that truncates.
bf16 results (8 significant bits) are off by at most 2^-8 relative each, so by no more in the norm."""
import pytest
import torch

import seq_helpers as H

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
F32_TOL, BF16_TOL = 1e-5, 2.0 ** -8


def _mat(seed, *shape, scale=1.0):
    return (torch.randn(*shape, generator=torch.Generator().manual_seed(seed)) * scale).bfloat16().to(DEV)


@pytest.fixture(scope="module")
def ops():
    from umbrella_b200 import _lib_seq, ops_seq
    yield ops_seq
    assert _lib_seq.load().umbs_kernel_timeouts() == 0


# one tile, its edges, several tiles per block; columns that leave 16-byte rows of C and columns that do not
@pytest.mark.parametrize("M,N,K", [(17, 8, 32), (128, 64, 64), (127, 65, 96), (129, 257, 64), (300, 1544, 1056), (64, 6144, 128),
                                   (2049, 513, 192), (1500, 3088, 256)])
def test_plain(ops, M, N, K):
    a, w = _mat(1, M, K), _mat(2, N, K)
    ref = a.double() @ w.double().T
    assert H.rel_err(ops.gemm(a, w, out_f32=True), ref.cpu()) < F32_TOL
    assert H.rel_err(ops.gemm(a, w), ref.cpu()) < BF16_TOL


def test_overlapping_rows_are_taken(ops):
    a, w = _mat(41, 1, 64), _mat(42, 40, 64)
    ref = a.double() @ w.double().T
    assert H.rel_err(ops.gemm(a.expand(33, 64), w, out_f32=True), ref.expand(33, 40).cpu()) < F32_TOL
    x = _mat(43, 600)                                            # row i starts at number 8 i
    rows = x.as_strided((60, 64), (8, 1))
    assert H.rel_err(ops.gemm(rows, w, out_f32=True), (rows.double() @ w.double().T).cpu()) < F32_TOL


def test_rows_are_bitwise_the_same_in_every_tile_width(ops):
    a, w = _mat(3, 2100, 512), _mat(4, 2048, 512)               # 17 x 8 tiles of 256 columns; 64 rows alone: tiles of 64
    full = ops.gemm(a, w, out_f32=True)
    assert torch.equal(ops.gemm(a[1030:1094].contiguous(), w, out_f32=True), full[1030:1094])
    assert torch.equal(ops.gemm(a[5:305].contiguous(), w, out_f32=True), full[5:305])


@pytest.mark.parametrize("M,N,K", [(40, 33, 64), (200, 128, 96), (1000, 1000, 64)])
def test_epilogues(ops, M, N, K):
    from umbrella_b200 import _lib_seq as S
    a, w, w2 = _mat(5, M, K), _mat(6, N, K, scale=K ** -0.5), _mat(7, 2 * N, K, scale=K ** -0.5)
    bias, gate = torch.randn(2 * N, device=DEV), torch.randn(M, N, device=DEV)
    z, z2 = a.double() @ w.double().T, a.double() @ w2.double().T
    got = ops.gemm_ex(a, w, out_f32=True, bias=bias, out_gate=gate)
    assert H.rel_err(got, ((z + bias[:N].double()) * torch.sigmoid(gate.double())).cpu()) < F32_TOL
    got = ops.gemm_ex(a, w2, out_f32=True, act=S.UMBS_ACT_SILU, bias=bias)
    g, u = (z2 + bias.double()).split(N, 1)
    assert H.rel_err(got, (torch.nn.functional.silu(g) * u).cpu()) < F32_TOL
    got = ops.gemm_unary(a, w, S.UMBS_UNARY_RELU2, out_f32=True, cols=N // 2)
    assert H.rel_err(got, torch.cat([z[:, :N // 2].clamp(min=0) ** 2, z[:, N // 2:]], 1).cpu()) < F32_TOL


@pytest.mark.parametrize("M,heads,n,k", [(33, 3, 48, 32), (260, 5, 128, 64), (130, 2, 320, 96)])
def test_batched_over_heads(ops, M, heads, n, k):
    a, w = _mat(8, M, heads * k), _mat(9, heads, n, k)
    ref = torch.einsum("mhk,hnk->mhn", a.double().view(M, heads, k), w.double())
    got = ops.gemm(a, w, out_f32=True, groups=heads, a_goff=k, c_goff=n + 2)     # (an odd place for every head's columns)
    assert H.rel_err(got.view(M, heads, n + 2)[..., :n], ref.cpu()) < F32_TOL
    gate = torch.randn(M, heads, device=DEV)
    got = ops.gemm_head_gate(a, w, gate, heads, n, k)
    assert H.rel_err(got, (ref * torch.sigmoid(gate.double())[..., None]).reshape(M, -1).cpu()) < BF16_TOL


@pytest.mark.parametrize("sizes", [(17, 0, 3, 128, 129), (0, 0, 300, 1, 0), (700, 650, 640, 660, 655)])
@pytest.mark.parametrize("K", [64, 160])
def test_rows_sorted_by_expert(ops, sizes, K):
    """Gathered rows with the gated activation, then the sorted rows themselves; groups without rows, of one row, of a tile and a row."""
    E, n, total = len(sizes), 96, sum(sizes)
    off = torch.tensor([0] + list(torch.tensor(sizes).cumsum(0)), dtype=torch.int32, device=DEV)
    T = max(max(sizes), 20)
    src = torch.randint(0, T, (total,), generator=torch.Generator().manual_seed(1)).to(torch.int32).to(DEV)
    h, gu, down = _mat(10, T, K), _mat(11, E, 2 * n, K, scale=K ** -0.5), _mat(12, E, 72, n, scale=n ** -0.5)
    y = ops.gemm(h, gu, groups=E, n=n, dual=True, limit=7.0, grp_off=off, row_src=src, rows=total, max_rows=T)
    o = ops.gemm(y, down, out_f32=True, groups=E, grp_off=off, rows=total, max_rows=T)
    at = 0
    for e, m in enumerate(sizes):
        if m == 0:
            continue
        z = h[src[at:at + m].long()].double() @ gu[e].double().T
        g, u = z[:, :n].clamp(max=7.0), z[:, n:].clamp(-7.0, 7.0)
        assert H.rel_err(y[at:at + m], (g * torch.sigmoid(1.702 * g) * (u + 1)).cpu()) < BF16_TOL
        assert H.rel_err(o[at:at + m], (y[at:at + m].double() @ down[e].double().T).cpu()) < F32_TOL
        at += m


@pytest.mark.parametrize("M,N,K", [(1, 1, 5), (63, 65, 17), (64, 64, 16), (65, 130, 100), (200, 31, 1000)])
@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
def test_true_32_bit_tiles(ops, M, N, K, dt):
    """The fp32 kernel (and what no tensor-core tile takes: K not a multiple of 32) at the edges of its 64 x 64 x 16 tiles, rows that no
    16-byte load may take, gated pairs."""
    g = torch.Generator().manual_seed(M)
    a, w = torch.randn(M, K + 1, generator=g).to(dt).to(DEV)[:, 1:], torch.randn(2 * N, K, generator=g).to(dt).to(DEV)
    z = a.double() @ w.double().T
    assert H.rel_err(ops.gemm(a, w, out_f32=True), z.cpu()) < 2e-6                        # sqrt(1000) 2^-24
    got = ops.gemm(a, w, n=N, dual=True, limit=7.0, out_f32=True)
    gate, up = z[:, :N].clamp(max=7.0), z[:, N:].clamp(-7.0, 7.0)
    assert H.rel_err(got, (gate * torch.sigmoid(1.702 * gate) * (up + 1)).cpu()) < 4e-6   # a product of two such sums


def test_groups_that_run_backwards_are_taken(ops):
    """A negative step between the groups' columns: no tensor map describes it."""
    x, w = _mat(51, 40, 3 * 64), _mat(52, 3, 48, 64)
    got = ops.gemm(x[:, 128:], w, out_f32=True, groups=3, a_goff=-64, c_goff=48)
    ref = torch.cat([x[:, 128 - 64 * i:192 - 64 * i].double() @ w[i].double().T for i in range(3)], 1)
    assert H.rel_err(got, ref.cpu()) < F32_TOL


@pytest.mark.parametrize("act", ["CLAMPED_GLU", "GELU_TANH", "SILU"])
@pytest.mark.parametrize("M", [17, 300])
def test_activations_are_those_of_the_fp32_kernels(ops, act, M):
    """Weight rows with a single one make every sum a bf16 number exactly, so the results show the activation alone.  They are those of
    the fp32 kernel bit for bit (a sigmoid below 2^-126 is 0 here and a subnormal number there: 1e-35 covers it times a number of the
    row), and within 1e-6 of float64 in the norm (a tanh or an exponential of two units in the last place, an argument rounded three
    times)."""
    from umbrella_b200 import _lib_seq as S
    K, N = 64, 32
    a = _mat(61, M, K, scale=3.0)
    a[0, :8] = torch.tensor([0.0, 1e-30, 88.0, -88.0, 100.0, -100.0, 3e38, -3e38], dtype=torch.bfloat16)
    w = torch.zeros(2 * N, K, dtype=torch.bfloat16, device=DEV)
    w[torch.arange(2 * N), torch.arange(2 * N) % K] = 1.0                 # gate n reads number n, up n reads number 32 + n
    run = lambda x, y: ops.gemm_ex(x, y, out_f32=True, act=getattr(S, "UMBS_ACT_" + act), limit=7.0)
    got, f32 = run(a, w), run(a.float(), w.float())
    assert bool(((got == f32) | ((got - f32).abs() < 1e-35)).all())
    g, u = a[1:, :N].double(), a[1:, N:].double()
    if act == "CLAMPED_GLU":
        g, u = g.clamp(max=7.0), u.clamp(-7.0, 7.0) + 1
    f = {"CLAMPED_GLU": lambda t: t * torch.sigmoid(1.702 * t), "SILU": torch.nn.functional.silu,
         "GELU_TANH": lambda t: torch.nn.functional.gelu(t, approximate="tanh")}[act]
    assert H.rel_err(got[1:], (f(g) * u).cpu()) < 1e-6


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_general_kernel_rows_have_the_same_bits_in_both_tile_heights(ops, dtype):
    """fp32 (and bf16 rows that nothing else takes: K = 66): tiles of 16 rows while tiles of 64 would not give every SM a block."""
    K, N = 66, 8200                                              # 129 blocks of columns: 64 rows are few, 128 are many
    a, w = (torch.randn(128, K, generator=torch.Generator().manual_seed(71)).to(dtype).to(DEV), torch.randn(2 * N, K, generator=torch.Generator().manual_seed(72)).to(dtype).to(DEV))
    full, dual = ops.gemm(a, w[:N], out_f32=True), ops.gemm(a, w[:4800], out_f32=True, dual=True, limit=7.0)      # (75 blocks of 32 pairs)
    assert H.rel_err(full, (a.double() @ w[:N].double().T).cpu()) < F32_TOL
    for lo, hi in ((0, 1), (3, 18), (5, 21), (7, 24), (60, 124)):
        assert torch.equal(ops.gemm(a[lo:hi].contiguous(), w[:N], out_f32=True), full[lo:hi])
        assert torch.equal(ops.gemm(a[lo:hi].contiguous(), w[:4800], out_f32=True, dual=True, limit=7.0), dual[lo:hi])
    x, v = a[:, :64].contiguous(), w[:48, :32].reshape(2, 24, 32).contiguous()               # groups, a step between them
    got = ops.gemm(x[:17], v, out_f32=True, groups=2, a_goff=32, c_goff=24)
    assert H.rel_err(got, torch.cat([x[:17, 32 * i:32 * i + 32].double() @ v[i].double().T for i in range(2)], 1).cpu()) < F32_TOL


# few rows: both forms (multiply-add: 32-bit; tensor core: tiles of 8 and of 16 weight rows, pieces of 16 and of 32 bytes), columns and k that end inside a tile, a piece, a warp's share.  A sum is rounded at most 24 times: pieces, lanes, warps.
@pytest.mark.parametrize("M", [1, 2, 3, 4, 5, 8, 9, 16])
@pytest.mark.parametrize("N,K", [(1, 8), (19, 40), (130, 520), (1030, 1032), (2050, 1304), (515, 4104)])
@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
def test_few_rows(ops, M, N, K, dt):
    a, w = _mat(51, M, K).to(dt), _mat(52, N, K).to(dt)
    if dt == torch.float32:
        a, w = a + 2.0 ** -9 * _mat(53, M, K).float(), w + 2.0 ** -9 * _mat(54, N, K).float()
    ref = a.double() @ w.double().T
    assert H.rel_err(ops.gemm(a, w, out_f32=True), ref.cpu()) < 24 * 2.0 ** -24
    assert H.rel_err(ops.gemm(a, w), ref.cpu()) < (BF16_TOL if dt == torch.bfloat16 else 24 * 2.0 ** -24)


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("K", [64, 1032, 2048])
def test_few_rows_sorted_by_expert(ops, dt, K):
    from umbrella_b200 import _lib_seq as S
    sizes, ff = (3, 0, 16, 1, 9), 37
    off = torch.tensor([0, 3, 3, 19, 20, 29], dtype=torch.int32, device=DEV)
    a, w = _mat(55, 40, K).to(dt), _mat(56, 5, 2 * ff, K, scale=K ** -0.5).to(dt)
    src = torch.randperm(40, generator=torch.Generator().manual_seed(57))[:29].int().to(DEV)
    got = ops.gemm(a, w, groups=5, n=ff, dual=True, limit=3.0, grp_off=off, row_src=src, rows=29, max_rows=16)
    lo = 0
    for g, n in enumerate(sizes):
        x = a[src[lo:lo + n].long()].double()
        gate, up = (x @ w[g, :ff].double().T).clamp(max=3.0), (x @ w[g, ff:].double().T).clamp(-3.0, 3.0)
        ref = gate * torch.sigmoid(1.702 * gate) * (up + 1)
        if n:
            assert H.rel_err(got[lo:lo + n], ref.cpu()) < (BF16_TOL if dt == torch.bfloat16 else 1e-6)
        lo += n


@pytest.mark.parametrize("N,K", [(100, 512), (1030, 2048), (6144, 1024)])
def test_few_rows_do_not_depend_on_the_others(ops, N, K):
    a, w = _mat(58, 16, K), _mat(59, N, K)
    full = ops.gemm(a, w, out_f32=True)
    for m in (1, 4, 8, 11):
        assert torch.equal(ops.gemm(a[:m].contiguous(), w, out_f32=True), full[:m])


# 32-bit operands as three bf16 parts: tiles of 128 rows and of 32 to 160 columns, k in steps of 64 (sums of two steps are added up), the
# edges of each.  A product's dropped terms are below 2^-25 of it; sums: 16 terms cut off 8 times in a row (2^-23 each at most), then
# K / 128 rounded additions; random signs: 1e-6 covers K = 1000.
F32_SPLIT_TOL = 1e-6


def _mat32(seed, *shape, scale=1.0):
    return (torch.randn(*shape, generator=torch.Generator().manual_seed(seed)) * scale).to(DEV)


def _kernel(dt, M, N, K, **kw):
    from umbrella_b200 import _lib_seq as S
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    return S.load().umbs_gemm_kernel(S.UMBS_F32 if dt == torch.float32 else S.UMBS_BF16, M, N, K, kw.get("groups", 1), kw.get("sorted", 0), kw.get("dual", 0), sms)


# (the first four sizes are few enough products for the streamed rows in some of the calls; the others take the tiles in all)
@pytest.mark.parametrize("M,N,K", [(128, 1028, 1000), (129, 1990, 68), (1200, 33, 516), (40, 9001, 64), (777, 513, 128), (300, 5000, 132),
                                   (70000, 2, 8), (128, 8300, 1000), (129, 19900, 68), (4200, 33, 516), (40, 41000, 64)])
def test_split_products(ops, M, N, K):
    from umbrella_b200 import _lib_seq as S
    if (M, N, K) not in ((128, 1028, 1000), (129, 1990, 68), (1200, 33, 516), (40, 9001, 64)):
        assert _kernel(torch.float32, M, N, K) == _kernel(torch.float32, M, N, K, dual=1) == S.UMBS_GEMM_SPLIT
    a, w = _mat32(81, M, K), _mat32(82, N, K)
    assert H.rel_err(ops.gemm(a, w), (a.double() @ w.double().T).cpu()) < F32_SPLIT_TOL
    w2, bias, gate = _mat32(83, 2 * N, K, scale=K ** -0.5), _mat32(84, 2 * N), _mat32(85, M, N)
    z = a.double() @ w2.double().T + bias.double()
    ref = torch.nn.functional.silu(z[:, :N]) * z[:, N:] * torch.sigmoid(gate.double())
    assert H.rel_err(ops.gemm_ex(a, w2, act=S.UMBS_ACT_SILU, bias=bias, out_gate=gate), ref.cpu()) < 2 * F32_SPLIT_TOL
    got = ops.gemm_unary(a, w2[:N].contiguous(), S.UMBS_UNARY_SILU, cols=N // 2)
    z = a.double() @ w2[:N].double().T
    assert H.rel_err(got, torch.cat([torch.nn.functional.silu(z[:, :N // 2]), z[:, N // 2:]], 1).cpu()) < 2 * F32_SPLIT_TOL


def test_split_products_sorted_by_expert(ops):
    sizes, ff, K = (130, 0, 3, 260, 1), 200, 196
    off = torch.tensor([0, 130, 130, 133, 393, 394], dtype=torch.int32, device=DEV)
    a, w = _mat32(86, 300, K), _mat32(87, 5, 2 * ff, K, scale=K ** -0.5)
    src = torch.randint(0, 300, (394,), generator=torch.Generator().manual_seed(88)).int().to(DEV)
    got = ops.gemm(a, w, groups=5, n=ff, dual=True, limit=3.0, grp_off=off, row_src=src, rows=394, max_rows=300)
    lo = 0
    for g, n in enumerate(sizes):
        x = a[src[lo:lo + n].long()].double()
        gate, up = (x @ w[g, :ff].double().T).clamp(max=3.0), (x @ w[g, ff:].double().T).clamp(-3.0, 3.0)
        if n:
            assert H.rel_err(got[lo:lo + n], (gate * torch.sigmoid(1.702 * gate) * (up + 1)).cpu()) < 2 * F32_SPLIT_TOL
        lo += n


def test_split_products_of_wider_rows_and_of_groups(ops):
    from umbrella_b200 import _lib_seq as S
    M, N, K = 400, 4000, 72
    assert _kernel(torch.float32, M, N, K) == S.UMBS_GEMM_SPLIT
    x, w = _mat32(93, M, K + 28), _mat32(94, N, K)
    a = x[:, 12:12 + K]                                              # rows further apart than they are long, from a 16-byte boundary on
    assert H.rel_err(ops.gemm(a, w), (a.double() @ w.double().T).cpu()) < F32_SPLIT_TOL
    heads, n, k = 3, 1500, 68
    assert _kernel(torch.float32, M, n, k, groups=heads) == S.UMBS_GEMM_SPLIT
    a, w = _mat32(95, M, heads * k), _mat32(96, heads, n, k)
    got = ops.gemm(a, w, groups=heads, a_goff=k, c_goff=n + 1)
    ref = torch.einsum("mhk,hnk->mhn", a.double().view(M, heads, k), w.double())
    assert H.rel_err(got.view(M, heads, n + 1)[..., :n], ref.cpu()) < F32_SPLIT_TOL
    assert bool((got.view(M, heads, n + 1)[..., n] == 0).all())


# Operands that three bf16 parts in fp32's own scale do not hold (below 2^-110), beside partners that lift the results back into range, on either
# side; results near and in the subnormal range: one rounding more, 2^-150 for an element.
@pytest.mark.parametrize("x,y", [(-118, 40), (-124, 60), (-126, 100), (-140, 110), (60, -118), (110, -140), (-60, -66), (-74, -66)])
def test_split_products_of_small_numbers_beside_large_ones(ops, x, y):
    from umbrella_b200 import _lib_seq as S
    M, N, K = 400, 4000, 64
    assert _kernel(torch.float32, M, N, K) == S.UMBS_GEMM_SPLIT
    a, w = _mat32(97, M, K) * 2.0 ** x, _mat32(98, N, K) * 2.0 ** y
    got, ref = ops.gemm(a, w).double(), a.double() @ w.double().T
    assert float((got - ref).norm() / ref.norm()) < F32_SPLIT_TOL + 2.0 ** -150 * (M * N) ** 0.5 / float(ref.norm())


def test_split_products_of_rows_far_apart(ops):
    """Gathered rows up to 64 GiB behind the first, where offsets of 32 bits in 16-byte pieces end."""
    from umbrella_b200 import _lib_seq as S
    ld, M, N, K = 2 ** 26, 60, 5000, 256
    if torch.cuda.mem_get_info()[0] < 80 << 30:
        pytest.skip("65 GiB of memory")
    assert _kernel(torch.float32, M, N, K) == S.UMBS_GEMM_SPLIT
    a, w, src = torch.empty(257 * ld, device=DEV).as_strided((257, K), (ld, 1)), _mat32(99, 1, N, K), torch.arange(256, 256 - 4 * M, -4, dtype=torch.int32, device=DEV)
    a.copy_(_mat32(100, 257, K))
    got = ops.gemm(a, w, grp_off=torch.tensor([0, M], dtype=torch.int32, device=DEV), row_src=src, rows=M, max_rows=M)
    assert H.rel_err(got, (a[src.long()].double() @ w[0].double().T).cpu()) < F32_SPLIT_TOL
    del a
    torch.cuda.empty_cache()


@pytest.mark.parametrize("value", [1e32, float("nan")])
def test_split_products_beyond_the_parts_on_every_tile(ops, value):
    """Several tiles a block, all of whose sums are worked out again, while the other warps wait for the next tile.  Tolerance: chains of 256
    rounded additions of random signs, sqrt(256) 2^-24 = 1e-6, three times."""
    from umbrella_b200 import _lib_seq as S
    M, N, K = 4100, 1610, 256
    assert _kernel(torch.float32, M, N, K) == S.UMBS_GEMM_SPLIT
    a, w = _mat32(77, M, K) * value, _mat32(78, N, K)
    got, ref = ops.gemm(a, w).double(), a.double() @ w.double().T
    if value == value:
        assert float((got - ref).norm() / ref.norm()) < 3e-6
    else:
        assert bool(torch.isnan(got).all())


@pytest.mark.parametrize("M,N", [(200, 2000), (400, 4000)])          # streamed, tiles
def test_split_products_of_numbers_at_the_ends_of_the_range(ops, M, N):
    """Infinite and NaN operands, numbers that round to infinity in bf16, and rows so small that their low parts vanish there."""
    from umbrella_b200 import _lib_seq as S
    K = 64
    assert _kernel(torch.float32, M, N, K) == (S.UMBS_GEMM_SPLIT if M == 400 else S.UMBS_GEMM_FEW_ROWS)
    a, w = _mat32(91, M, K), _mat32(92, N, K)
    a[0, 3], a[1, 5], a[2, 7], w[9, 11] = float("inf"), float("nan"), 3.4e38, float("-inf")
    a[3], w[10] = a[3] * 2.0 ** -120, w[10] * 2.0 ** -100
    w[:, 7] = w[:, 7] * 2.0 ** -20                                   # (the sums of row 2 stay in range)
    got, ref = ops.gemm(a, w), a.double() @ w.double().T
    fin = torch.isfinite(ref.float())
    assert torch.equal(torch.isfinite(got), fin) and torch.equal(torch.isnan(got), torch.isnan(ref))
    assert torch.equal(got[~fin & ~torch.isnan(ref)], ref[~fin & ~torch.isnan(ref)].float())
    keep = torch.ones(N, dtype=torch.bool, device=DEV)
    keep[9] = False
    for rows in (slice(2, 3), slice(3, 4), slice(4, M)):
        x, y = got[rows][:, keep].double(), ref[rows][:, keep]
        assert ((x - y).norm() / y.norm()).item() < F32_SPLIT_TOL
    x, y = got[4:, 10].double(), ref[4:, 10]
    assert ((x - y).norm() / y.norm()).item() < F32_SPLIT_TOL


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("K,max_rows", [(64, 200), (64, 16), (40, 200)])          # tensor-core tiles, few rows, neither
def test_sorted_rows_of_no_group_are_zero(ops, dt, K, max_rows):
    """Rows behind the last group's, into memory that something else has used; a_goff is not used by sorted rows."""
    sizes = (9, 0, 13)
    off = torch.tensor([0, 9, 9, 22], dtype=torch.int32, device=DEV)
    a, w = _mat(101, 30, K).to(dt), _mat(102, 3, 50, K).to(dt)
    junk = [torch.full((30, 50), float("nan"), device=DEV) for _ in range(8)]
    del junk
    got = ops.gemm(a, w, groups=3, grp_off=off, rows=30, max_rows=max_rows, out_f32=True)
    assert bool((got[22:] == 0).all())
    lo = 0
    for g, n in enumerate(sizes):
        if n:
            assert H.rel_err(got[lo:lo + n], (a[lo:lo + n].double() @ w[g].double().T).cpu()) < F32_TOL
        lo += n


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("K,max_rows", [(64, 200), (64, 16), (40, 200)])          # tensor-core tiles, few rows, neither
@pytest.mark.parametrize("f32", [True, False])
def test_sorted_rows_in_front_of_the_first_group_are_zero(ops, dt, K, max_rows, f32):
    """A slice of the experts: the offsets begin behind rows of others."""
    from umbrella_b200 import _lib_seq as S
    off = torch.tensor([5, 9, 9, 22], dtype=torch.int32, device=DEV)
    a, w = _mat(103, 30, K).to(dt), _mat(104, 3, 50, K).to(dt)
    got = torch.full((30, 50), float("nan"), dtype=torch.float32 if f32 else dt, device=DEV)
    S.check(S.load().umbs_gemm_sorted(ops._mode(a), a.data_ptr(), K, w.data_ptr(), K, 50 * K, got.data_ptr(), 50, int(f32), max_rows, 30, 50, K, 3,
                                      off.data_ptr(), None, 0, 0.0, ops._stream()), "gemm")
    assert bool((got[:5] == 0).all()) and bool((got[22:] == 0).all())
    tol = F32_TOL if got.dtype == torch.float32 else BF16_TOL
    for g, (lo, hi) in enumerate([(5, 9), (9, 9), (9, 22)]):
        if hi > lo:
            assert H.rel_err(got[lo:hi], (a[lo:hi].double() @ w[g].double().T).cpu()) < tol


# pairs of SMs: tiles of 256 rows x 256 columns (gate|up: 128 of each), rows and columns that end in either half; groups
@pytest.mark.parametrize("M,N,K", [(1000, 3100, 1056), (1537, 2049, 64), (4096, 1100, 96), (1290, 6144, 512)])
def test_pairs_of_blocks(ops, M, N, K):
    from umbrella_b200 import _lib_seq as S
    a, w, w2 = _mat(111, M, K), _mat(112, N, K), _mat(113, 2 * N, K, scale=K ** -0.5)
    ref = a.double() @ w.double().T
    got = ops.gemm(a, w, out_f32=True)
    assert H.rel_err(got, ref.cpu()) < F32_TOL
    assert H.rel_err(ops.gemm(a, w), ref.cpu()) < BF16_TOL
    assert torch.equal(ops.gemm(a[-100:].contiguous(), w, out_f32=True), got[-100:])              # (single blocks)
    bias = torch.randn(2 * N, device=DEV)
    z = a.double() @ w2.double().T + bias.double()
    ref = torch.nn.functional.silu(z[:, :N]) * z[:, N:]
    assert H.rel_err(ops.gemm_ex(a, w2, act=S.UMBS_ACT_SILU, bias=bias, out_f32=True), ref.cpu()) < F32_TOL


# sizes for which the rule takes pairs in every call: one, two and several steps of 64 of k, k that ends inside one, an odd number of
# columns, last tiles with rows in the first block alone
@pytest.mark.parametrize("M,N,K,dual", [(1000, 3100, 1056, 0), (6000, 6145, 64, 0), (4200, 4099, 128, 0), (1100, 4098, 736, 0),
                                        (1290, 6144, 512, 1), (2900, 3071, 96, 1), (6000, 3071, 64, 1)])
def test_products_that_take_pairs(ops, M, N, K, dual):
    from umbrella_b200 import _lib_seq as S
    assert _kernel(torch.bfloat16, M, N, K, dual=dual) == S.UMBS_GEMM_PAIRS
    assert _kernel(torch.bfloat16, 100, N, K, dual=dual) != S.UMBS_GEMM_PAIRS
    a, w = _mat(116, M, K), _mat(117, N * (1 + dual), K, scale=K ** -0.5)
    bias = torch.randn(w.shape[0], device=DEV)
    run = lambda x, f32: ops.gemm_ex(x, w, act=S.UMBS_ACT_SILU if dual else 0, bias=bias, out_f32=f32)
    ref = a.double() @ w.double().T + bias.double()
    if dual:
        ref = torch.nn.functional.silu(ref[:, :N]) * ref[:, N:]
    got = run(a, True)
    assert H.rel_err(got, ref.cpu()) < F32_TOL
    assert H.rel_err(run(a, False), ref.cpu()) < BF16_TOL
    assert torch.equal(run(a[-100:].contiguous(), True), got[-100:])                              # (single blocks)


@pytest.mark.parametrize("M,heads,n,k", [(700, 5, 520, 128), (1290, 3, 1550, 1056)])             # single blocks, pairs
@pytest.mark.parametrize("gap", [0, 1])
def test_pairs_of_blocks_over_heads(ops, M, heads, n, k, gap):
    from umbrella_b200 import _lib_seq as S
    assert (_kernel(torch.bfloat16, M, n, k, groups=heads) == S.UMBS_GEMM_PAIRS) == (M == 1290)
    a, w = _mat(114, M, heads * k), _mat(115, heads, n, k)
    ref = torch.einsum("mhk,hnk->mhn", a.double().view(M, heads, k), w.double())
    got = ops.gemm(a, w, out_f32=True, groups=heads, a_goff=k, c_goff=n + gap).view(M, heads, n + gap)
    assert H.rel_err(got[..., :n], ref.cpu()) < F32_TOL
    assert bool((got[..., n:] == 0).all())
