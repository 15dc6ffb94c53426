"""Each kernel schedule of the attention forward at the sizes where it can go wrong: the last CTA of
the first wave, one item more than there are slots, the borders of the dispatch rule (plan_fwd in
csrc/fa_b200_api.cu), groups of heads that do not divide evenly, many rounds of taking items over.

Every result has to be bit for bit what the same head gives alone (where one CTA per tile runs, or
one CTA), and sampled heads are held to the CPU oracle at the tolerances of test_parity_gpu.py."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _heads_near(items, tiles):
    return max(1, -(-items // tiles))


def _slots():
    return 2 * torch.cuda.get_device_properties(0).multi_processor_count


def _launched(call):
    """What `call` launches, from a graph that it is captured into (and never run): the one kernel's name, as the compiler
    writes it, and the bytes of shared memory that a CTA of it asks for."""
    import ctypes

    class Node(ctypes.Structure):                # CUDA_KERNEL_NODE_PARAMS_v2
        _fields_ = [("func", ctypes.c_void_p), ("grid", ctypes.c_uint * 3), ("block", ctypes.c_uint * 3), ("smem", ctypes.c_uint),
                    ("params", ctypes.c_void_p), ("extra", ctypes.c_void_p), ("kern", ctypes.c_void_p), ("ctx", ctypes.c_void_p)]

    call()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        call()
    cu, n, nodes = ctypes.CDLL("libcuda.so.1"), ctypes.c_size_t(8), (ctypes.c_void_p * 8)()
    assert cu.cuGraphGetNodes(ctypes.c_void_p(graph.raw_cuda_graph()), nodes, ctypes.byref(n)) == 0 and n.value == 1
    node, name = Node(), ctypes.c_char_p()
    assert cu.cuGraphKernelNodeGetParams_v2(ctypes.c_void_p(nodes[0]), ctypes.byref(node)) == 0
    assert (cu.cuFuncGetName(ctypes.byref(name), ctypes.c_void_p(node.func)) if node.func else
            cu.cuKernelGetName(ctypes.byref(name), ctypes.c_void_p(node.kern))) == 0
    return name.value.decode(), node.smem


@pytest.mark.parametrize("B,H,N", [(1, 1, 400), (1, 12, 512), (1, 24, 700), (1, 12, 1500), (1, 1, 16384)])
@pytest.mark.parametrize("causal", [True, False])
def test_few_tiles_share_an_sm_with_another_streams(fa_lib, B, H, N, causal):
    """Calls of at most a tile per SM leave room on every SM for a CTA of another stream's attention call, as all others
    do: two calls that overlap then take 0.57 to 0.67 of the time that they take one after the other."""
    from tfg_flashattention_b200 import custom_flash_attn as cfa
    q = torch.zeros(B, H, N, 64, device="cuda", dtype=torch.bfloat16)
    assert B * H * -(-N // 128) <= _slots() // 2
    out = torch.empty_like(q)
    name, smem = _launched(lambda: cfa.forward(q, q, q, causal=causal, out=out))
    assert "fa_fwd" in name
    most = torch.cuda.get_device_properties(0).shared_memory_per_multiprocessor
    assert 2 * (smem + 1024) <= most             # (1 KB of each CTA's is the system's)


@pytest.mark.parametrize("N,items", [
    (128, "slots"), (128, "slots+1"), (90, "3*slots"),              # one K/V tile: one item / static
    (300, "slots+3"), (500, "2*slots-4"), (512, "2*slots"),         # up to four: static, then dynamic
    (700, "4*slots//3-6"), (700, "4*slots//3+6"), (1024, "5*slots"),
    (2048, "2*slots"), (2177, "2*slots"),                            # dynamic
])
@pytest.mark.parametrize("causal", [True, False])
def test_schedule_borders(fa_lib, N, items, causal):
    from oracle.attention_oracle import manual_attention
    from tfg_flashattention_b200 import custom_flash_attn as cfa
    tiles = -(-N // 128)
    heads = _heads_near(eval(items, {"slots": _slots()}), tiles)
    g = torch.Generator(device="cuda").manual_seed(N + heads)
    q, k, v = (torch.randn(1, heads, N, 64, device="cuda", generator=g).bfloat16() for _ in range(3))
    o = torch.full_like(q, float("nan"))
    _, lse = cfa.forward(q, k, v, causal=causal, return_lse=True, out=o)
    assert cfa.last_status() == 0
    assert torch.isfinite(o).all() and torch.isfinite(lse).all()
    for h in {0, 1 % heads, heads // 2, heads - 1}:
        one = (t[:, h:h + 1].contiguous() for t in (q, k, v))
        alone, alone_lse = cfa.forward(*one, causal=causal, return_lse=True)
        assert torch.equal(alone[0, 0], o[0, h]) and torch.equal(alone_lse[0, 0], lse[0, h])
    h = heads - 1
    ref, ref_lse = manual_attention(*(t[:, h:h + 1].float().cpu() for t in (q, k, v)), causal=causal, return_lse=True)
    d = (o[0, h].float().cpu() - ref[0, 0]).abs()
    assert d.max().item() <= 2e-2 and d.mean().item() <= 2e-3
    assert ((lse[0, h].cpu() - ref_lse[0, 0]).abs() <= 1e-3 * ref_lse[0, 0].abs().clamp_min(1.0)).all()


@pytest.mark.parametrize("N", [384, 385, 512, 513, 640, 900])
@pytest.mark.parametrize("causal", [True, False])
def test_a_tile_per_sm_at_most(fa_lib, N, causal):
    """The largest grid of at most a tile per SM, one head more, and a grid of several waves give the same bits, with key
    rows that make the running maximum jump, from other strides too."""
    from tfg_flashattention_b200 import custom_flash_attn as cfa
    sms, tiles = _slots() // 2, -(-N // 128)
    most = sms // tiles
    g = torch.Generator(device="cuda").manual_seed(N)
    qkv = torch.randn(1, N, 3, 5 * most, 64, device="cuda", generator=g).bfloat16()
    qkv[:, ::37, 1] *= 6
    q, k, v = (qkv[:, :, i].transpose(1, 2) for i in range(3))
    want, want_lse = cfa.forward(q, k, v, causal=causal, return_lse=True)
    for heads in (1, most, most + 1):
        part = [t[:, 2:2 + heads] for t in (q, k, v)]
        o, lse = cfa.forward(*part, causal=causal, return_lse=True, out=torch.full((1, heads, N, 64), float("nan"), device="cuda", dtype=q.dtype))
        assert cfa.last_status() == 0
        assert torch.equal(o, want[:, 2:2 + heads]) and torch.equal(lse, want_lse[:, 2:2 + heads])


@pytest.mark.parametrize("items", ["2*slots-2", "2*slots", "2*slots+2", "21*slots//10-2", "21*slots//10+2", "30*slots//11", "30*slots//11+4"])
@pytest.mark.parametrize("causal", [True, False])
def test_two_tiles_above_two_rounds(fa_lib, items, causal):
    """Two K/V tiles: dealt to the resident CTAs up to 2.7 rounds, taken over above."""
    from tfg_flashattention_b200 import custom_flash_attn as cfa
    heads = eval(items, {"slots": _slots()}) // 2
    g = torch.Generator(device="cuda").manual_seed(heads)
    q, k, v = (torch.randn(1, heads, 200, 64, device="cuda", generator=g).bfloat16() for _ in range(3))
    inside = 11 * 2 * heads <= 30 * _slots()
    assert cfa.plan(q, k, v, causal=causal) == (("static", _slots()) if inside else ("dynamic", 2 * heads))
    o = cfa.forward(q, k, v, causal=causal, out=torch.full_like(q, float("nan")))
    assert cfa.last_status() == 0 and torch.isfinite(o).all()
    for h in (0, heads // 2, heads - 1):
        assert torch.equal(cfa.forward(*(t[:, h:h + 1].contiguous() for t in (q, k, v)), causal=causal)[0, 0], o[0, h])


@pytest.mark.parametrize("N,heads", [(12287, 3), (12288, 3), (12300, 3), (12416, 6)])      # the border; one CTA per tile, taken over
def test_long_causal_rows_are_those_of_a_shorter_sequence(fa_lib, N, heads):
    """Long causal sequences have the diagonal tile behind the tile loop: row for row the bits of the same rows in a
    sequence that has it inside.  Which of the two is launched: fa_fwd_kernel's template arguments (schedule, causal, ragged,
    long)."""
    from tfg_flashattention_b200 import custom_flash_attn as cfa
    g = torch.Generator(device="cuda").manual_seed(N)
    q, k, v = (torch.randn(1, heads, N, 64, device="cuda", generator=g).bfloat16() for _ in range(3))
    k[:, :, ::701] *= 5
    o, lse = cfa.forward(q, k, v, return_lse=True, out=torch.full_like(q, float("nan")))
    assert cfa.last_status() == 0 and torch.isfinite(o).all() and torch.isfinite(lse).all()
    one_item = cfa.plan(q, k, v)[0] == "cta_per_tile"
    assert one_item == (heads == 3)
    name, _ = _launched(lambda: cfa.forward(q, k, v, out=torch.empty_like(q)))
    assert f"fa_fwd_kernelILi{0 if one_item else 2}ELb1ELb0ELb{int(N >= 12288)}EEEv" in name
    short, short_lse = cfa.forward(q[:, :, :12200], k[:, :, :12200], v[:, :, :12200], return_lse=True)
    assert torch.equal(o[:, :, :12200], short) and torch.equal(lse[:, :, :12200], short_lse)


def test_order_by_groups_of_heads(fa_lib):
    """32 MB of K and V (N * 256 bytes a head) are ordered together, 15 heads of 8200 rows: 33 heads make
    three groups of 11, 34 groups of 12, 12 and 10."""
    from tfg_flashattention_b200 import custom_flash_attn as cfa
    for heads, N in ((33, 8200), (34, 8200)):
        g = torch.Generator(device="cuda").manual_seed(heads)
        q, k, v = (torch.randn(1, heads, N, 64, device="cuda", generator=g).bfloat16() for _ in range(3))
        o = cfa.forward(q, k, v, out=torch.full_like(q, float("nan")))
        assert cfa.last_status() == 0 and torch.isfinite(o).all()
        for h in (0, 14, 15, 16, heads - 1):
            assert torch.equal(cfa.forward(*(t[:, h:h + 1].contiguous() for t in (q, k, v)))[0, 0], o[0, h])


@pytest.mark.parametrize("B,N", [(32, 1024), (12, 1100)])
def test_taking_over_while_the_first_wave_waits(fa_lib, B, N):
    """Part of the resident slots are held by another stream's kernel, so that running CTAs take over CTAs
    of the first wave, whose items are not those of their block index (the mirror in fa_fwd_sm100.cuh).
    The other kernel: 128 tiles of one head, 16384 rows, one per SM, about 150 us."""
    from tfg_flashattention_b200 import custom_flash_attn as cfa
    g = torch.Generator(device="cuda").manual_seed(N)
    q, k, v = (torch.randn(B, 25, N, 64, device="cuda", generator=g).bfloat16() for _ in range(3))
    long = torch.randn(1, 1, 16384, 64, device="cuda", generator=g).bfloat16()
    want, want_lse = cfa.forward(q, k, v, return_lse=True)
    held, side = torch.empty_like(long), torch.cuda.Stream()
    torch.cuda.synchronize()
    for _ in range(4):
        o = torch.full_like(q, float("nan"))
        torch.cuda.synchronize()
        with torch.cuda.stream(side):
            cfa.forward(long, long, long, causal=False, out=held)
        _, lse = cfa.forward(q, k, v, return_lse=True, out=o)
        torch.cuda.synchronize()
        assert cfa.last_status() == 0
        assert torch.equal(o, want) and torch.equal(lse, want_lse)


def test_captured_launches_depend_early_only_on_the_librarys_own(fa_lib):
    """In a graph, an edge of programmatic dependent launch between two of the library's kernels, a plain one
    behind any other; two captures in a row; replays give what the calls give."""
    import ctypes
    from tfg_flashattention_b200 import block_ops
    from tfg_flashattention_b200 import custom_flash_attn as cfa
    g = torch.Generator(device="cuda").manual_seed(3)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
    x, scale, shift, q = rnd(8, 256), rnd(256), rnd(256), rnd(1, 4, 300, 64)

    def work():
        a = x + 1
        b = block_ops.add_layernorm(a, None, scale, shift)                  # behind torch's
        c = block_ops.add_layernorm(b, None, scale, shift)                  # behind ours
        d = cfa.forward(q, q, q)                                            # ours
        e = cfa.forward(d, d, d)                                            # ours
        f = e + 1
        return c, f, cfa.decode(f[:, :, 0].contiguous(), f, f, 300)         # behind torch's

    want = work()
    for _ in range(2):
        graph = torch.cuda.CUDAGraph(keep_graph=True)
        with torch.cuda.graph(graph):
            got = work()
        n = ctypes.c_size_t(64)
        nodes, data = (ctypes.c_void_p * 64)(), (ctypes.c_uint8 * 8 * 64)()        # CUgraphEdgeData: ports, type, padding
        assert ctypes.CDLL("libcuda.so.1").cuGraphGetEdges_v2(ctypes.c_void_p(graph.raw_cuda_graph()), nodes, (ctypes.c_void_p * 64)(),
                                                              data, ctypes.byref(n)) == 0
        assert sum(data[i][2] == 1 for i in range(n.value)) == 3 and n.value >= 6   # 1: CU_GRAPH_DEPENDENCY_TYPE_PROGRAMMATIC
        graph.instantiate()
        for t in got:
            t.zero_()
        graph.replay()
        assert all(torch.equal(a, b) for a, b in zip(got, want))
