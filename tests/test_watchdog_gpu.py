"""A bounded wait that runs out: the kernel reports it and returns, and the context stays usable.

Every mbarrier wait in the attention kernel has a time limit; when one runs out the kernel writes
a code to a status word, every role drains and leaves through the normal exit, and
fa_b200_last_status hands the code to the host (the reference has nothing of the kind: its
cudaGetLastError result is dropped, src/cpp/torch_bind.cpp:34-39).  To see that path run, a second
build of the library (-DFA_WAIT_TEST) shortens the limit to 2 ms and has the TMA producer leave out
the second K tile, whose barrier is then armed by nobody -- a flag that nothing sets.  No trap, no
bad address, no endless loop: the launch ends by itself within a few tens of milliseconds.
"""
import ctypes
import time

import pytest
import torch

pytestmark = pytest.mark.gpu

WATCHDOG_BASE = 0x10000
# The missing K tile stalls three waits at once: the issuer's for that tile (2), and behind it the
# producer's for the Q slot (9) and the softmax warps' for the next S (4).  They started within a
# microsecond or two of each other, so which one runs out first -- and gets to write the word -- is
# a matter of that microsecond; any of the three is the right report.
EXPECTED_WAITS = {2: b"K/V tile load", 9: b"Q slot", 4: b"S = QK^T"}
# The 96 CTAs of a long sequence, one tile each: the producer has more to load and stops at the slot of V 0 instead (3).
EXPECTED_WAITS_LONG = {2: b"K/V tile load", 3: b"K/V slot", 4: b"S = QK^T"}


@pytest.mark.parametrize("N,product,test_build,expected", [
    # two causal tiles; the test build runs them as one CTA, whose first item needs two K tiles
    (256, ("cta_per_tile", 2), ("static", 1), EXPECTED_WAITS),
    # the form with the diagonal tile behind the tile loop; every CTA but the first tile's needs the missing K tile
    (12288, ("cta_per_tile", 96), ("cta_per_tile", 96), EXPECTED_WAITS_LONG),
])
def test_wait_runs_out_is_reported_and_the_next_launch_is_correct(fa_lib, N, product, test_build, expected):
    if not torch.cuda.is_available():
        pytest.fail("GPU tests need a CUDA device")
    from tfg_flashattention_b200 import _lib, build
    from tfg_flashattention_b200 import custom_flash_attn as cfa
    wt = ctypes.CDLL(build.build_wait_test_library())
    wt.fa_b200_fwd.argtypes = [ctypes.POINTER(_lib.FaParams)]
    wt.fa_b200_fwd.restype = ctypes.c_int
    wt.fa_b200_last_status.argtypes = [ctypes.c_int, ctypes.c_void_p]
    wt.fa_b200_last_status.restype = ctypes.c_int
    wt.fa_b200_strerror.argtypes = [ctypes.c_int]
    wt.fa_b200_strerror.restype = ctypes.c_char_p

    torch.manual_seed(3)
    q, k, v = (torch.randn(1, 1, N, 64, device="cuda").bfloat16() for _ in range(3))
    assert cfa.plan(q, k, v) == product
    schedule, grid = ctypes.c_int32(-1), ctypes.c_int32(0)
    params = cfa._fwd_params(q, k, v, q, None, True, None)
    wt.fa_b200_fwd_plan.argtypes = [ctypes.POINTER(_lib.FaParams), ctypes.POINTER(ctypes.c_int32), ctypes.POINTER(ctypes.c_int32)]
    assert wt.fa_b200_fwd_plan(ctypes.byref(params), ctypes.byref(schedule), ctypes.byref(grid)) == 0
    assert (_lib.SCHEDULES[schedule.value], grid.value) == test_build
    good = cfa.forward(q, k, v)
    assert cfa.last_status() == 0

    o = torch.empty_like(q)
    p = cfa._fwd_params(q, k, v, o, None, True, None)
    stream = torch.cuda.current_stream().cuda_stream
    t0 = time.perf_counter()
    assert wt.fa_b200_fwd(ctypes.byref(p)) == 0          # the launch itself succeeds
    code = wt.fa_b200_last_status(0, stream)             # synchronises: the kernel has returned
    elapsed = time.perf_counter() - t0
    assert code & ~0xff == WATCHDOG_BASE and (code & 0xff) in expected, hex(code)
    message = wt.fa_b200_strerror(code)
    assert b"watchdog" in message and expected[code & 0xff] in message
    assert elapsed < 2.0, f"the kernel took {elapsed:.2f} s to give up"
    assert wt.fa_b200_last_status(0, stream) == 0        # reading the word cleared it

    # the context is intact: the product library computes the same bits as before
    again = cfa.forward(q, k, v)
    assert cfa.last_status() == 0
    assert torch.equal(again, good)


@pytest.mark.parametrize("B,pos", [(1, 5), (1, 900), (8, 70)])
def test_step_gives_up_and_the_next_one_is_correct(fa_lib, monkeypatch, B, pos):
    """The generation step: the test build's block 0 keeps back its words of the embedding, so that every block
    waits for them until its wait runs out; the weight stream then waits for ring slots that nobody gives
    back.  All of them give up, the launch returns, the workspace is made ready again."""
    from types import SimpleNamespace

    from tfg_flashattention_b200 import _lib, build, gpt2, step
    from tfg_flashattention_b200 import custom_flash_attn as cfa
    wt = ctypes.CDLL(build.build_wait_test_library())
    for name in ("fa_b200_gpt_step", "fa_b200_last_status", "fa_b200_strerror"):
        getattr(wt, name).argtypes, getattr(wt, name).restype = getattr(fa_lib, name).argtypes, getattr(fa_lib, name).restype

    cfg = {"vocab_size": 503, "context_length": 1024, "emb_dim": 768, "n_heads": 12, "n_layers": 2, "drop_rate": 0.0,
           "qkv_bias": True, "impl_type": "cuda"}
    model = gpt2.init_random(gpt2.GPTModel(cfg, dtype=torch.bfloat16), seed=2).cuda().eval().prepare_for_inference()
    ids = torch.randint(0, 503, (B, pos + 1), device="cuda")
    caches = model.allocate_kv_cache(B, 1024)
    with torch.no_grad():
        model(ids[:, :pos], kv_caches=caches, pos=0)
    plan = model._step_plan
    workspace = plan.new_workspace(B)
    good = model._step(ids[:, pos:], caches, pos, workspace=workspace)
    assert good is not None and cfa.last_status() == 0

    after = torch.full((B,), -1, dtype=torch.long, device="cuda")
    scratch = [tuple(t.clone() for t in pair) for pair in caches]
    t0 = time.perf_counter()
    with monkeypatch.context() as m:
        m.setattr(step, "_lib", SimpleNamespace(load=lambda: wt, FaGptStepParams=_lib.FaGptStepParams, strerror=_lib.strerror))
        assert plan.step(ids[:, pos:], scratch, pos, workspace=workspace, next_ids=after) is not None      # launched
    stream = torch.cuda.current_stream().cuda_stream
    code = wt.fa_b200_last_status(0, stream)
    elapsed = time.perf_counter() - t0
    assert code & ~0xff == WATCHDOG_BASE and (code & 0xff) in (17, 18, 19), hex(code)
    assert b"generation step" in wt.fa_b200_strerror(code)
    assert elapsed < 2.0, f"the kernel took {elapsed:.2f} s to give up"
    assert wt.fa_b200_last_status(0, stream) == 0
    for new, old in zip(scratch, caches):              # no cached row but the step's own was written
        for a, b in zip(new, old):
            keep = torch.arange(1024, device="cuda") != pos
            assert torch.equal(a[:, keep], b[:, keep])

    # whoever asks for the status of the library that gave up gets its workspaces back in order
    with monkeypatch.context() as m:
        m.setattr(cfa, "_lib", SimpleNamespace(load=lambda: SimpleNamespace(fa_b200_last_status=lambda *a: code),
                                               WATCHDOG_BASE=_lib.WATCHDOG_BASE))
        workspace.fill_(1)
        assert cfa.last_status() == code and (workspace == 0).all()
    again = model._step(ids[:, pos:], caches, pos, workspace=workspace)
    assert cfa.last_status() == 0 and torch.equal(again, good)
