"""Decode attention against a 64-bit restatement: every number of heads per KV head, contexts around the edges of the
16 positions of a step, splits that leave some CTAs without positions, and caches whose rows past the position hold NaN."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _tables(S):
    inv = 1.0 / (10000.0 ** (torch.arange(0, 128, 2, device="cuda").float() / 128))
    ang = torch.arange(S, device="cuda").float()[:, None] * inv[None]
    return ang.cos().contiguous(), ang.sin().contiguous()


def _rope(x, cos, sin):
    a, b = x[..., :64], x[..., 64:]
    return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)


def _run(qkv, kc, vc, pos, cos, sin, nh, nkv, nsplit):
    import torch_ccl_b200._C as C

    B = qkv.shape[0]
    out = torch.full((B, nh * 128), 7.0, device="cuda", dtype=torch.bfloat16)
    scratch = torch.zeros(C.decode_attention_scratch_bytes(B, nh, nsplit) // 4 + 1, device="cuda")
    counters = torch.zeros(B * nh, device="cuda", dtype=torch.int32)
    C.decode_attention(qkv, kc, vc, pos, cos, sin, out, scratch, counters, nh, nkv, nsplit)
    assert (counters == 0).all()
    return out


@pytest.mark.parametrize("nh,nkv", [(2, 2), (4, 2), (6, 2), (4, 1), (10, 2), (12, 2), (8, 1)])
@pytest.mark.parametrize("nsplit", [1, 2, 5])
def test_against_64_bits(nh, nkv, nsplit):
    at = [0, 1, 14, 15, 16, 17, 31, 32, 33, 95, 96, 97, 160, 299]
    B, S = len(at), 300
    g = torch.Generator(device="cuda").manual_seed(nh * 100 + nkv * 10 + nsplit)
    qkv = torch.randn(B, (nh + 2 * nkv) * 128, generator=g, device="cuda").bfloat16()
    kc, vc = (torch.randn(B, nkv, S, 128, generator=g, device="cuda").bfloat16() for _ in range(2))
    pos = torch.tensor(at, device="cuda", dtype=torch.int32)
    for i, p in enumerate(at):
        kc[i, :, p:], vc[i, :, p:] = float("nan"), float("nan")
    cos, sin = _tables(S)
    k0, v0 = kc.clone(), vc.clone()
    out = _run(qkv, kc, vc, pos, cos, sin, nh, nkv, nsplit).double().view(B, nh, 128)
    x = qkv.view(B, -1, 128)
    for i, p in enumerate(at):
        new_k = _rope(x[i, nh:nh + nkv].double(), cos[p].double(), sin[p].double())
        # one rounding to bf16; the 32-bit rotation may fall on the other side of a tie
        assert ((kc[i, :, p].double() - new_k).abs() <= new_k.abs() * 2.0**-8 + 1e-6).all()
        assert torch.equal(vc[i, :, p], x[i, nh + nkv:])
        for c, c0 in ((kc, k0), (vc, v0)):
            assert torch.equal(c[i, :, :p], c0[i, :, :p]) and torch.isnan(c[i, :, p + 1:].float()).all()
        q = _rope(x[i, :nh].double(), cos[p].double(), sin[p].double()) / 128**0.5
        k, v = (c[i, :, : p + 1].double().repeat_interleave(nh // nkv, 0) for c in (kc, vc))
        w = torch.softmax(torch.einsum("hd,htd->ht", q, k), -1)
        ref = torch.einsum("ht,htd->hd", w, v)
        # half a bf16 unit in the last place is at most 2^-8 of the value; scores of a few units and their exponentials carry
        # a few 2^-22 each, which the sum of |w v| scales
        bound = ref.abs() * 2.0**-8 + torch.einsum("ht,htd->hd", w, v.abs()) * 2.0**-17
        assert ((out[i] - ref).abs() <= bound).all(), (nh, nkv, nsplit, p)


def test_infinite_values():
    """An infinite V element gives an infinite output in its dim only."""
    nh, nkv, S = 4, 2, 64
    qkv = torch.ones(1, (nh + 2 * nkv) * 128, device="cuda").bfloat16()
    kc, vc = torch.ones(1, nkv, S, 128, device="cuda").bfloat16(), torch.ones(1, nkv, S, 128, device="cuda").bfloat16()
    vc[0, 0, 3, 5] = float("inf")
    cos, sin = torch.ones(S, 64, device="cuda"), torch.zeros(S, 64, device="cuda")
    for nsplit in (1, 2):
        out = _run(qkv, kc.clone(), vc.clone(), torch.tensor([40], device="cuda", dtype=torch.int32), cos, sin, nh, nkv, nsplit).view(nh, 128)
        want = torch.ones(nh, 128, device="cuda").bfloat16()
        want[:2, 5] = float("inf")
        assert torch.equal(out, want)


def test_position_outside_the_cache():
    nh, nkv, S = 8, 2, 32
    qkv = torch.randn(2, (nh + 2 * nkv) * 128, device="cuda").bfloat16()
    kc, vc = (torch.randn(2, nkv, S, 128, device="cuda").bfloat16() for _ in range(2))
    k0, v0 = kc.clone(), vc.clone()
    out = _run(qkv, kc, vc, torch.tensor([-1, S], device="cuda", dtype=torch.int32), *_tables(S), nh, nkv, 3)
    assert (out == 0).all() and torch.equal(kc, k0) and torch.equal(vc, v0)
