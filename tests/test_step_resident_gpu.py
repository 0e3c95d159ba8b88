"""One-sequence decode steps as a resident grid (csrc/step_resident.cu) against the chain of launches that serves every other step: the same operations in
the same order, so the same bits in every vector, cache row and logit."""
import pytest
import torch

from mistralrs_b200 import mmq, model as M

pytestmark = pytest.mark.gpu

SHAPES = {      # width, inner, heads, KV heads, head size
    "gqa4": (2560, 1536, 16, 4, 128),         # ten blocks a row: a span and a part of one
    "mha": (2560, 2816, 16, 16, 128),         # one query head a KV head, nine tiles at most; 176 and 80 blocks of Q8_0 a row
    "gqa2_64": (3072, 512, 32, 16, 64),
    "gqa7": (3584, 1024, 28, 4, 128),         # heads that do not fill the warps' groups; Q6_K rows off 16-byte boundaries
    "gqa8_64": (2560, 768, 64, 8, 64),
}


def _pair(cuda, monkeypatch, shape, quant, dtype, layers=1, neox=True, block=16, vocab=1001, types=None, ctx=700):
    hidden, inter, heads, kv, dim = SHAPES[shape]
    if types is not None:
        monkeypatch.setattr(M, "tensor_type", types)
    cfg = M.LlamaConfig.tiny_test(quant=quant, n_layers=layers, hidden=hidden, inter=inter, n_heads=heads, n_kv_heads=kv, head_dim=dim, vocab=vocab,
                                  rope_neox=neox, block_size=block, max_pos=4096, synth_scale_exp=(-15.5, -14.5))
    w = M.LlamaWeights(cfg, cuda, dtype=dtype, fast_synth=True)
    resident, chain = (M.LlamaRunner(w, batch=1, max_ctx=ctx) for _ in range(2))
    chain.step_struct.extension = M.STEP_Q8
    g = torch.Generator(device="cuda").manual_seed(5)
    for a, b in zip(resident.k_cache + resident.v_cache, chain.k_cache + chain.v_cache):
        a.copy_(torch.randn(a.shape, device="cuda", generator=g))
        b.copy_(a)
    return resident, chain


def _ran_resident(run):
    """Tiles leave their sums in the scratch of the resident grid; nothing else writes there."""
    return bool(run.resident[256:].any())


def _launches(run, at):
    """Kernels of one step, counted on a captured one: the grid's are one for 32 layers (and the embedding, the argmax, the advance)."""
    import bench
    run.reset(at)
    g = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(g):
        run.step()
    return bench.count_graph_kernels(g)


def _step(run, at, token=11):
    run.reset(at)
    run.set_tokens([token])
    run.step()
    torch.cuda.synchronize()
    return {k: run.buf[k].clone() for k in ("q", "k", "v", "attn_out", "x2", "act", "x", "logits", "out_token")}


def _same(resident, chain, at):
    a, b = _step(resident, at), _step(chain, at)
    assert bool(torch.isfinite(b["logits"].float()).all()) and bool(b["logits"].any())
    for k in a:
        assert torch.equal(a[k], b[k]), (at, k, float((a[k].double() - b[k].double()).norm() / b[k].double().norm()))
    assert all(torch.equal(x, y) for x, y in zip(resident.k_cache + resident.v_cache, chain.k_cache + chain.v_cache)), at


@pytest.mark.parametrize("ctx", [60, 500, 1500])
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("quant,dtype", [("q4_k_m", torch.float16), ("q8_0", torch.bfloat16)])
def test_step_equals_chain(cuda, monkeypatch, shape, quant, dtype, ctx):
    """One tile a head (which leaves nothing in the scratch: the launches tell), up to eight (a cluster's sums) and more (rounded partial results);
    contexts around a warp's, a step's and a tile's tokens."""
    resident, chain = _pair(cuda, monkeypatch, shape, quant, dtype, neox=shape != "gqa4", ctx=ctx)
    for at in (0, 1, 15, 16, 59, 63, 64, 65, 127, 128, 200, 497, 640, 1499):
        if at < ctx:
            _same(resident, chain, at)
    assert resident.is_resident() and not chain.is_resident()
    assert _ran_resident(resident) == (resident.padded_tiles > 1) and not _ran_resident(chain)
    assert _launches(resident, 1) == 4 < _launches(chain, 1)


@pytest.mark.parametrize("shape,dtype", [("gqa4", torch.bfloat16), ("gqa7", torch.float16)])
def test_more_tiles_than_a_warp_has_lanes(cuda, monkeypatch, shape, dtype):
    """From the 33rd tile on a lane holds two tiles' states: on both sides of it, of a tile's end and of the context's."""
    resident, chain = _pair(cuda, monkeypatch, shape, "q4_k_m", dtype, ctx=37 * 64)
    assert resident.is_resident() and resident.padded_tiles > 33
    tile = resident.split_pages * resident.cfg.block_size
    for at in (31 * tile, 32 * tile - 2, 32 * tile - 1, 32 * tile, 32 * tile + 1, 33 * tile - 1, 33 * tile, 2200, 37 * 64 - 1):
        _same(resident, chain, at)
    assert _ran_resident(resident)


def test_two_runners_on_two_streams(cuda, monkeypatch):
    """Grids that each want all SMs, from graphs on streams of their own, beside a third stream's products: they run one after the other, with their bits."""
    a, b = _pair(cuda, monkeypatch, "gqa4", "q4_k_m", torch.bfloat16, layers=2)
    b.step_struct.extension = M.STEP_RESIDENT
    for run in (a, b):
        run.capture()
    for x, y in zip(a.k_cache + a.v_cache, b.k_cache + b.v_cache):
        y.copy_(x)

    def start():
        for run, token in ((a, 7), (b, 8)):
            run.reset(60)
            run.set_tokens([token])
        torch.cuda.synchronize()

    start()
    for run in (a, b):
        for _ in range(60):
            run.replay()
        torch.cuda.synchronize()
    want = [(run.logits().clone(), [t.clone() for t in run.k_cache + run.v_cache]) for run in (a, b)]
    start()
    streams, m = [torch.cuda.Stream() for _ in range(3)], torch.randn(2048, 2048, device=cuda, dtype=torch.bfloat16)
    torch.cuda.synchronize()
    for i in range(60):
        for run, stream in zip((a, b), streams):
            with torch.cuda.stream(stream):
                run.replay()
        with torch.cuda.stream(streams[2]):
            m @ m
    torch.cuda.synchronize()
    mmq.check_timeouts(cuda)
    for run, (logits, caches) in zip((a, b), want):
        assert torch.equal(run.logits(), logits) and all(torch.equal(x, y) for x, y in zip(run.k_cache + run.v_cache, caches))


@pytest.mark.parametrize("block", [8, 24, 32])
def test_types_a_matrix_and_page_sizes(cuda, monkeypatch, block):
    """q and k in Q6_K, v in Q8_0, o_proj in Q6_K, gate and up in Q8_0, down in Q4_K, the head in Q6_K with an odd number of rows; pages of other sizes."""
    kinds = {"attn_q": "q6_k", "attn_k": "q6_k", "attn_v": "q8_0", "attn_output": "q6_k", "ffn_gate": "q8_0", "ffn_up": "q8_0", "output": "q6_k"}
    resident, chain = _pair(cuda, monkeypatch, "gqa4", "q4_k_m", torch.float16, block=block, types=lambda cfg, name, layer=0: kinds.get(name, "q4_k"))
    for at in (5, 100, 501):
        _same(resident, chain, at)
    assert _ran_resident(resident)


def test_generation_in_a_graph(cuda, monkeypatch):
    """Replays follow one another as eager steps do, bit for bit, and leave the words of the grid's barriers as they were."""
    eager, graph = _pair(cuda, monkeypatch, "gqa4", "q4_k_m", torch.bfloat16, layers=2)
    graph.step_struct.extension = M.STEP_RESIDENT
    graph.capture()
    for a, b in zip(eager.k_cache + eager.v_cache, graph.k_cache + graph.v_cache):      # (the capture's warm-up step wrote position 0)
        b.copy_(a)
    for run in (eager, graph):
        run.reset(60)
        run.set_tokens([7])
    for _ in range(40):
        eager.step()
        graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(eager.logits(), graph.logits())
    assert all(torch.equal(a, b) for a, b in zip(eager.k_cache + eager.v_cache, graph.k_cache + graph.v_cache))
    assert not bool(graph.resident[:256].any()) and _ran_resident(graph)


def test_more_layers_than_a_launch_holds(cuda, monkeypatch):
    resident, chain = _pair(cuda, monkeypatch, "gqa2_64", "q4_k_m", torch.bfloat16, layers=33)
    _same(resident, chain, 100)
    assert _ran_resident(resident)


def test_what_the_grid_declines(cuda, monkeypatch):
    """Other block types, long tiles, a scratch that is too small, the measuring switches: the chain, by its bits and its launches.  (A sequence at the end of its
    context stays on the grid, by the chain's rules.)"""
    resident, chain = _pair(cuda, monkeypatch, "gqa4", "q4_k_m", torch.float16, types=lambda cfg, name, layer=0: "q4_0" if name == "ffn_down" else "q4_k")
    assert torch.equal(_step(resident, 100)["logits"], _step(chain, 100)["logits"]) and not _ran_resident(resident)
    monkeypatch.undo()
    for shape, ctx, grid in (("gqa8_64", 9 * 1024, True), ("gqa8_64", 10 * 1024, False), ("gqa2_64", 2304, True), ("gqa2_64", 2512, False), ("mha", 4096, True)):
        resident, chain = _pair(cuda, monkeypatch, shape, "q4_k_m", torch.float16, ctx=ctx)       # tokens x KV heads a tile: 64 for each element of a head
        assert resident.is_resident() == grid, (shape, ctx)
        _same(resident, chain, 300)
        assert _ran_resident(resident) == grid
    resident, chain = _pair(cuda, monkeypatch, "gqa4", "q4_k_m", torch.float16, ctx=160)
    resident.step_struct.resident_bytes -= 16
    assert torch.equal(_step(resident, 50)["logits"], _step(chain, 50)["logits"]) and not _ran_resident(resident)
    resident.step_struct.resident_bytes += 16
    for mask in (1, 2):
        assert resident.is_resident()
        for run in (resident, chain):
            run.step_struct.skip_mask = mask
        assert not resident.is_resident() and _launches(resident, 50) == _launches(chain, 50) and not _ran_resident(resident)
        for run in (resident, chain):
            run.step_struct.skip_mask = 0
    before = [t.clone() for t in resident.k_cache + resident.v_cache]
    resident.context_lens.fill_(160)          # full: attends, writes no cache row, sets the flag
    resident.step()
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(before, resident.k_cache + resident.v_cache))
    assert int(resident.error_flag.item()) & 1 and _ran_resident(resident)
    assert bool(torch.isfinite(resident.logits().float()).all())


def test_steps_go_on_as_a_chain_once_a_wait_has_run_out(cuda, monkeypatch):
    """The device's word, set here by the host: eager steps are the chain's and leave the scratch alone, replays of a resident grid are refused, and a
    step that is captured then is a chain."""
    resident, chain = _pair(cuda, monkeypatch, "gqa4", "q4_k_m", torch.float16)
    resident.capture()
    chain.capture()                          # (a capture's warm-up step writes position 0)
    assert resident.is_resident() and not chain.is_resident()
    flag = mmq.timeout_word(cuda)
    try:
        flag[0] = 1
        scratch = resident.resident.clone()
        _same(resident, chain, 100)
        assert torch.equal(resident.resident, scratch) and not resident.is_resident()
        with pytest.raises(RuntimeError, match="ran out"):
            resident.replay()
        chain.reset(101)
        chain.replay()                       # (no kernel of this graph knows the word)
        resident.capture()
        chain.capture()
        for run in (resident, chain):
            run.reset(120)
            run.set_tokens([5])
            run.replay()
        torch.cuda.synchronize()
        assert torch.equal(resident.logits(), chain.logits()) and torch.equal(resident.resident, scratch)
    finally:
        flag[0] = 0
    assert resident.is_resident()


@pytest.mark.parametrize("layers", [1, 33])
def test_a_lost_grid_stays_lost(cuda, monkeypatch, layers):
    """What a grid whose wait ran out leaves in its scratch, put there by the host: launches with it, replays and eager ones, end at their first meeting with
    NaN for logits, no cache row written and the device's word set, in one launch and in two; zeroed, the scratch serves again."""
    run, _ = _pair(cuda, monkeypatch, "gqa2_64", "q4_k_m", torch.bfloat16, layers=layers)
    run.capture()

    def replay():
        run.reset(100)
        run.set_tokens([9])
        run.replay()
        torch.cuda.synchronize()
        return run.logits().clone()

    want, flag = replay(), mmq.timeout_word(cuda)
    word = run.resident[:4].view(torch.int32)
    assert bool(torch.isfinite(want.float()).all()) and int(word) == 0 and flag[0] == 0
    caches = [t.clone() for t in run.k_cache + run.v_cache]
    try:
        word.fill_(-2 ** 31)
        for launch in (run.replay, run.step, run.replay):
            flag[0] = 0                      # (only then does a call reach the grid)
            run.reset(200)
            run.set_tokens([9])
            run.logits().zero_()
            launch()
            torch.cuda.synchronize()
            assert flag[0] == 1 and int(word) == -2 ** 31
            assert bool(torch.isnan(run.logits()).all()) and 0 <= int(run.meta["token_ids"][0]) < run.cfg.vocab
            assert all(torch.equal(a, b) for a, b in zip(caches, run.k_cache + run.v_cache))
        with pytest.raises(RuntimeError, match="ran out"):
            run.replay()
        with pytest.raises(RuntimeError, match="ran out"):
            run.check_overflow()
    finally:
        flag[0] = 0
        run.resident[:256].zero_()
    assert torch.equal(replay(), want) and int(word) == 0
