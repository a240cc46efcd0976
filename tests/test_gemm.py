"""Numerics of the tcgen05 bf16 GEMM against a plain fp32 PyTorch reference."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _C():
    import torch_ccl_b200._C as C

    return C


def _ref(a, b):
    return a.float() @ b.float().t()


def _check(out, ref, k):
    tol = 2e-2 * (k ** 0.5) * 0.05 + 1e-2
    err = (out.float() - ref).abs().max().item()
    scale = ref.abs().max().item() + 1e-6
    assert err <= 1e-2 * scale + tol * 0.1, f"max err {err} (scale {scale})"


@pytest.mark.parametrize("M,N,K,bn", [
    (128, 16, 64, 16), (128, 16, 256, 16), (256, 128, 512, 128), (300, 72, 328, 0),
    (1024, 256, 4096, 256), (512, 64, 1024, 64), (128, 32, 2048, 32),
])
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
def test_gemm_plain(M, N, K, bn, out_dtype):
    torch.manual_seed(0)
    a = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
    b = torch.randn(N, K, device="cuda", dtype=torch.bfloat16)
    out = torch.empty(M, N, device="cuda", dtype=out_dtype)
    _C().gemm_bf16_tn(a, b, out, False, 0, 1, bn)
    torch.cuda.synchronize()
    _check(out, _ref(a, b), K)


@pytest.mark.parametrize("batch", [1, 4, 16])
@pytest.mark.parametrize("splitk", [1, 2, 4, 8, 16, 0])
def test_gemm_swap_ab_splitk(batch, splitk):
    """Decode shape: weights on the UMMA M side, the few activation rows on the N side."""
    torch.manual_seed(1)
    n_out, K = 1536, 4096
    w = torch.randn(n_out, K, device="cuda", dtype=torch.bfloat16) * 0.05
    x = torch.randn(batch, K, device="cuda", dtype=torch.bfloat16)
    out = torch.empty(batch, n_out, device="cuda", dtype=torch.bfloat16)
    _C().gemm_bf16_tn(w, x, out, True, 0, splitk, 16)
    torch.cuda.synchronize()
    _check(out, _ref(x, w), K)


@pytest.mark.parametrize("splitk", [1, 2, 4, 16])
def test_gemm_dual_swiglu(splitk):
    torch.manual_seed(2)
    inter, K, batch = 1376, 4096, 16
    w = torch.randn(2 * inter, K, device="cuda", dtype=torch.bfloat16) * 0.03
    x = torch.randn(batch, K, device="cuda", dtype=torch.bfloat16)
    out = torch.empty(batch, inter, device="cuda", dtype=torch.bfloat16)
    _C().gemm_bf16_tn(w, x, out, True, inter, splitk, 16)
    torch.cuda.synchronize()
    g = x.float() @ w[:inter].float().t()
    u = x.float() @ w[inter:].float().t()
    ref = torch.nn.functional.silu(g) * u
    _check(out, ref, K)


@pytest.mark.parametrize("M,N,K,bn", [(2048, 2560, 512, 128), (4096, 2560, 320, 256), (2000, 2500, 328, 128),
                                      (3000, 3100, 1032, 256), (8192, 4096, 4096, 0)])
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
def test_gemm_persistent(M, N, K, bn, out_dtype):
    """Large row-major results without a split (CTA pairs, walking a list of tiles): ordinary widths, ragged sizes."""
    torch.manual_seed(3)
    a = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
    b = torch.randn(N, K, device="cuda", dtype=torch.bfloat16)
    out = torch.empty(M, N, device="cuda", dtype=out_dtype)
    _C().gemm_bf16_tn(a, b, out, False, 0, 1, bn)
    torch.cuda.synchronize()
    _check(out, _ref(a, b), K)


@pytest.mark.parametrize("rows,K,batch", [(1536, 4096, 16), (1000, 1376, 5), (4096, 512, 16), (4096, 1376, 130)])
@pytest.mark.parametrize("splitk", [0, 1, 3, 16])
def test_gemm_pretiled_weights(rows, K, batch, splitk):
    """Weights packed as contiguous 128x64 tiles (ops.pack_weight), rows / K padded with zeros."""
    from torch_ccl_b200.ops import pack_weight, unpack_weight

    torch.manual_seed(4)
    w = torch.randn(rows, K, device="cuda", dtype=torch.bfloat16) * 0.05
    x = torch.randn(batch, K, device="cuda", dtype=torch.bfloat16)
    packed = pack_weight(w)
    assert torch.equal(unpack_weight(packed, rows, K), w)
    out = torch.empty(batch, rows, device="cuda", dtype=torch.bfloat16)
    bn = 16 if batch <= 16 else 128
    _C().gemm_bf16_tn(packed, x, out, True, 0, 1 if bn == 128 else splitk, bn, rows)
    torch.cuda.synchronize()
    _check(out, _ref(x, w), K)


@pytest.mark.parametrize("batch", [16, 200])
def test_gemm_pretiled_swiglu(batch):
    from torch_ccl_b200.ops import pack_weight

    torch.manual_seed(5)
    inter, K = 1376, 4096
    wg = torch.randn(inter, K, device="cuda", dtype=torch.bfloat16) * 0.03
    wu = torch.randn(inter, K, device="cuda", dtype=torch.bfloat16) * 0.03
    x = torch.randn(batch, K, device="cuda", dtype=torch.bfloat16)
    packed = torch.cat([pack_weight(wg), pack_weight(wu)])
    pad = (inter + 127) // 128 * 128
    out = torch.empty(batch, inter, device="cuda", dtype=torch.bfloat16)
    bn = 16 if batch <= 16 else 128
    _C().gemm_bf16_tn(packed, x, out, True, pad, 0 if bn == 16 else 1, bn, inter)
    torch.cuda.synchronize()
    ref = torch.nn.functional.silu(x.float() @ wg.float().t()) * (x.float() @ wu.float().t())
    _check(out, ref, K)


@pytest.mark.parametrize("M,N,K,width", [
    (129, 64, 64, 0),        # one row more than the one-CTA kernel takes, a single K step
    (256, 32, 72, 64),       # fewer columns than a tile, K not a multiple of the stage
    (385, 513, 448, 0),      # odd CTA of the last pair without rows; one column in the last tile, unaligned rows
    (1000, 1003, 520, 128),  # row starts that no TMA store can take
    (2049, 2500, 328, 96), (2049, 2500, 328, 160), (2049, 2500, 328, 224),
    (5000, 4100, 1032, 256),  # several tiles per pair: both accumulators, the ring across tiles
])
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
def test_gemm_cta_pairs(M, N, K, width, out_dtype):
    """Row-major results of more than 128 rows: 256-row tiles on CTA pairs, every tile width and both ways of storing."""
    torch.manual_seed(6)
    a = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
    b = torch.randn(N, K, device="cuda", dtype=torch.bfloat16)
    out = torch.full((M + 1, N), float("nan"), device="cuda", dtype=out_dtype)
    _C().gemm_bf16_tn(a, b, out[:M], False, 0, 1, width)
    torch.cuda.synchronize()
    ref = _ref(a, b)
    # fp32 sums of exact products in another order: K * 2^-24 of the largest partial sum; bf16 results: half a unit (2^-9)
    rel = K * 2.0**-24 + (2.0**-9 if out_dtype == torch.bfloat16 else 0.0)
    assert ((out[:M].float() - ref).norm() / ref.norm()).item() <= rel
    assert torch.isnan(out[M]).all(), "stored past the last row"


@pytest.mark.parametrize("rows,K,tokens", [(64, 64, 129), (1000, 1376, 257), (1536, 512, 1030)])
@pytest.mark.parametrize("dual", [False, True])
def test_gemm_cta_pairs_packed(rows, K, tokens, dual):
    """Pre-tiled weights as the B operand of the CTA-pair kernel, alone and as SwiGLU pairs."""
    from torch_ccl_b200.ops import pack_weight

    torch.manual_seed(7)
    w = [torch.randn(rows, K, device="cuda", dtype=torch.bfloat16) * 0.05 for _ in range(2)]
    x = torch.randn(tokens, K, device="cuda", dtype=torch.bfloat16)
    out = torch.full((tokens, rows), float("nan"), device="cuda", dtype=torch.bfloat16)
    if dual:
        _C().gemm_bf16_tn(torch.cat([pack_weight(t) for t in w]), x, out, True, (rows + 127) // 128 * 128, 1, 0, rows)
        ref = torch.nn.functional.silu(_ref(x, w[0])) * _ref(x, w[1])
    else:
        _C().gemm_bf16_tn(pack_weight(w[0]), x, out, True, 0, 1, 0, rows)
        ref = _ref(x, w[0])
    torch.cuda.synchronize()
    assert ((out.float() - ref).norm() / ref.norm()).item() <= 2.0**-9 + K * 2.0**-22  # silu's __expf adds 2 ulp


@pytest.mark.parametrize("rows,K,tokens", [(1000, 328, 300), (1504, 512, 1030)])  # gate and up rows that no tile divides
@pytest.mark.parametrize("width", [0, 64, 128])
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
def test_gemm_cta_pairs_swiglu_rows(rows, K, tokens, width, out_dtype):
    """SwiGLU over plain stacked gate and up rows as the B operand of the CTA-pair kernel: the odd CTA's rows start anywhere,
    and a given width counts the columns of each half."""
    torch.manual_seed(9)
    w = torch.randn(2 * rows, K, device="cuda", dtype=torch.bfloat16) * 0.05
    x = torch.randn(tokens, K, device="cuda", dtype=torch.bfloat16)
    out = torch.full((tokens + 1, rows), float("nan"), device="cuda", dtype=out_dtype)
    _C().gemm_bf16_tn(w, x, out[:tokens], True, rows, 1, width)
    torch.cuda.synchronize()
    ref = torch.nn.functional.silu(_ref(x, w[:rows])) * _ref(x, w[rows:])
    rel = K * 2.0**-22 + (2.0**-9 if out_dtype == torch.bfloat16 else 0.0)  # silu's __expf adds 2 ulp
    assert ((out[:tokens].float() - ref).norm() / ref.norm()).item() <= rel
    assert torch.isnan(out[tokens]).all(), "stored past the last row"


@pytest.mark.parametrize("M,N,K,width,split", [(256, 32, 16384, 32, 16), (4096, 16, 8192, 16, 8), (300, 64, 4096, 64, 4), (130, 17, 64, 32, 1)])
def test_gemm_narrow_results_split_k(M, N, K, width, split):
    """More than 128 rows but at most 64 columns: narrow tiles, K split over a cluster (the sums say which kernel it was)."""
    torch.manual_seed(8)
    a = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
    b = torch.randn(N, K, device="cuda", dtype=torch.bfloat16)
    auto, given = (torch.empty(M, N, device="cuda") for _ in range(2))
    _C().gemm_bf16_tn(a, b, auto)
    _C().gemm_bf16_tn(a, b, given, False, 0, split, width)
    assert torch.equal(auto, given)
    ref = _ref(a, b)
    assert ((auto - ref).norm() / ref.norm()).item() <= K * 2.0**-24


@pytest.mark.parametrize("M,N,K", [(300, 128, 256), (16, 128, 256), (300, 16, 1024)])
def test_gemm_behind_a_late_kernel(M, N, K):
    """A GEMM starts early and waits for the kernel before it, which may itself wait for a peer for longer than the GEMM's own
    waits are allowed to take (here: two and a half seconds, for a peer that does not exist)."""
    C = _C()
    c = C.CudaComm.emulated(2, 1 << 20, 2500, 1)
    a = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
    b = torch.randn(N, K, device="cuda", dtype=torch.bfloat16)
    out = torch.empty(M, N, device="cuda")
    C.gemm_bf16_tn(a, b, out)
    want = out.clone()
    out.fill_(float("nan"))
    torch.cuda.synchronize()
    C.emu_missing_peer_probe(c)
    C.gemm_bf16_tn(a, b, out)
    torch.cuda.synchronize()
    assert c.status()[0] == 1
    assert torch.equal(out, want)
