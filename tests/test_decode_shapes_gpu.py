"""Every launch shape of the decode kernel (decode_shape in csrc/fa_b200_api.cu): clusters of 1 to 16
CTAs, 128 to 512 threads, at the borders of the rule and of a CTA's rows (four rows per lane group and
step), against attention of the same bf16 numbers in fp64.

The kernel rounds once, to bf16: 8 significant bits, so at most 2^-8 of the value.  Its fp32 sums over
n <= 4100 rows of values up to about 5 and the exponentials (2^-22) add well under 1e-3 of their scale;
the part that is left where terms cancel is covered by 1e-4 absolute."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _close(o, want):
    return ((o.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-4).all()


@pytest.mark.parametrize("B,H,kv", [
    (1, 1, 1), (1, 3, 31), (1, 12, 95), (1, 12, 96), (2, 12, 191), (1, 25, 193), (4, 25, 383),   # clusters 1, 2, 4
    (1, 25, 767), (1, 25, 769), (2, 25, 1025),                                                    # 8, 16
    (1, 12, 1024), (1, 12, 1025), (1, 25, 2049), (1, 25, 4096), (1, 12, 2049), (1, 12, 4100),     # 256, 512 threads
    (41, 25, 64), (41, 25, 300), (42, 25, 300), (20, 25, 130), (21, 25, 777),                     # around 1036 heads, 518
])
@pytest.mark.parametrize("append", [False, True])
def test_decode_shapes(fa_lib, B, H, kv, append):
    from tfg_flashattention_b200 import custom_flash_attn as cfa
    g = torch.Generator(device="cuda").manual_seed(B * 100003 + H * 1009 + kv)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
    rows = kv + 5
    q, k, v = rnd(B, H, 64), rnd(B, rows, H, 64).transpose(1, 2), rnd(B, H, rows, 64)
    kn, vn = rnd(B, H, 64), rnd(B, H, 64)
    k_ref, v_ref = k.clone(), v.clone()
    if append:
        k_ref[:, :, kv - 1], v_ref[:, :, kv - 1] = kn, vn
    new = dict(k_new=kn, v_new=vn) if append else {}
    o, lse = cfa.decode(q, k, v, kv, return_lse=True, **new)
    assert torch.equal(k, k_ref) and torch.equal(v, v_ref)
    s = torch.einsum("bhd,bhnd->bhn", q.double(), k_ref[:, :, :kv].double()) / 8.0
    want = torch.einsum("bhn,bhnd->bhd", torch.softmax(s, -1), v_ref[:, :, :kv].double())
    assert _close(o, want)
    assert (lse.double() - torch.logsumexp(s, -1)).abs().max().item() <= 1e-4
    # a device length inside a launch sized for the whole cache: some CTAs then have few rows or none
    for n in {1, max(1, kv // 3), kv}:
        o2 = cfa.decode(q, k, v, torch.full((1,), n, dtype=torch.int32, device="cuda"))
        s = torch.einsum("bhd,bhnd->bhn", q.double(), k[:, :, :n].double()) / 8.0
        want = torch.einsum("bhn,bhnd->bhd", torch.softmax(s, -1), v[:, :, :n].double())
        assert _close(o2, want)


def test_more_heads_than_a_grid_dimension_of_65535(fa_lib):
    from tfg_flashattention_b200 import custom_flash_attn as cfa
    B, H = 70000, 1
    g = torch.Generator(device="cuda").manual_seed(1)
    q, k, v = (torch.randn(*s, device="cuda", generator=g).bfloat16() for s in ((B, H, 64), (B, H, 2, 64), (B, H, 2, 64)))
    o = cfa.decode(q, k, v, 2)
    s = torch.einsum("bhd,bhnd->bhn", q.double(), k.double()) / 8.0
    want = torch.einsum("bhn,bhnd->bhd", torch.softmax(s, -1), v.double())
    assert _close(o, want)


@pytest.mark.parametrize("B,H,kv", [(1, 3, 1), (1, 12, 95), (1, 25, 1025), (1, 12, 4100), (41, 25, 64)])
def test_scores_far_below_zero(fa_lib, B, H, kv):
    """Scores of about -1e33 (with LSE of that size), all equal but one in three: a softmax like any other.
    The smallest is not as small as an empty lane group's maximum."""
    from tfg_flashattention_b200 import custom_flash_attn as cfa
    g = torch.Generator(device="cuda").manual_seed(kv)
    q = torch.full((B, H, 64), 1e16, device="cuda").bfloat16()
    k = torch.full((B, H, kv, 64), -1e16, device="cuda").bfloat16()
    k[:, :, 1::3] *= 2
    v = torch.randn(B, H, kv, 64, device="cuda", generator=g).bfloat16()
    o, lse = cfa.decode(q, k, v, kv, return_lse=True)
    s = torch.einsum("bhd,bhnd->bhn", q.double(), k.double()) / 8.0
    want = torch.einsum("bhn,bhnd->bhd", torch.softmax(s, -1), v.double())
    assert s.max().item() < -1e32 and _close(o, want)
    assert ((lse.double() / torch.logsumexp(s, -1) - 1).abs() <= 1e-5).all()


def test_length_written_by_the_kernel_in_front(fa_lib):
    """A device length that is advanced between back-to-back launches, and a LayerNorm whose scale is."""
    from tfg_flashattention_b200 import block_ops
    from tfg_flashattention_b200 import custom_flash_attn as cfa
    g = torch.Generator(device="cuda").manual_seed(5)
    q, k, v = (torch.randn(*s, device="cuda", generator=g).bfloat16() for s in ((1, 4, 64), (1, 4, 64, 64), (1, 4, 64, 64)))
    x = torch.randn(8, 768, device="cuda", generator=g).bfloat16()
    n, scale, shift = torch.zeros(1, dtype=torch.int32, device="cuda"), torch.zeros(768, device="cuda").bfloat16(), torch.zeros(768, device="cuda").bfloat16()
    outs, norms = [], []
    for _ in range(64):
        n.add_(1)
        outs.append(cfa.decode(q, k, v, n))
        scale.add_(1)
        norms.append(block_ops.add_layernorm(x, None, scale, shift))
    for i in range(64):
        assert torch.equal(outs[i], cfa.decode(q, k, v, i + 1))
        assert torch.equal(norms[i], block_ops.add_layernorm(x, None, torch.full_like(scale, i + 1), shift))


@pytest.mark.parametrize("binding", ["ext", "ctypes"])
def test_rows_of_longer_tensors(fa_lib, torch_binding, binding):
    """out, k_new and v_new of [B, H, n, 64] stand for their first rows, through both bindings."""
    if binding == "ext" and torch_binding is None:
        pytest.skip("the torch extension binding could not be built here")
    from tfg_flashattention_b200 import custom_flash_attn as cfa
    g = torch.Generator(device="cuda").manual_seed(9)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
    q, k, v, kn, vn = rnd(2, 3, 1, 64), rnd(2, 3, 9, 64), rnd(2, 3, 9, 64), rnd(2, 3, 4, 64), rnd(2, 3, 4, 64)
    want = cfa.decode(q, k.clone(), v.clone(), 7, k_new=kn[:, :, 0].contiguous(), v_new=vn[:, :, 0].contiguous())
    cfa.set_binding(binding)
    try:
        out = torch.zeros(2, 3, 5, 64, dtype=torch.bfloat16, device="cuda")
        got = cfa.decode(q, k, v, 7, out=out, k_new=kn, v_new=vn)
    finally:
        cfa.set_binding("auto")
    assert got is out and torch.equal(out[:, :, :1], want) and (out[:, :, 1:] == 0).all()
    assert torch.equal(k[:, :, 6], kn[:, :, 0]) and torch.equal(v[:, :, 6], vn[:, :, 0])
