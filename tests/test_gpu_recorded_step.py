"""The recorded single-token step of the Qwen3 decoder against the same calls issued one by one: same kernels on the same
operands, so logits are equal to the last bit, whatever changes between two steps."""
import dataclasses

import pytest
import torch

pytestmark = pytest.mark.gpu
bf16 = torch.bfloat16
B, T, STEPS = 3, 20, 7


@pytest.fixture
def served():
    from omegalax_b200.parallel import mesh as mesh_lib
    from omegalax_b200.text import api

    mesh_lib.set_default_mesh(None)
    cfg = dataclasses.replace(api.resolve_config("Qwen/Qwen3-8B"), num_layers=2, emb_dim=256, mlp_dim=512, num_heads=4,
                              num_kv_heads=2, vocab_size=1024)
    model, cfg = api.init_model(cfg, 0, tp_size=1, fsdp_size=1, dp_size=1, device="cuda", dtype=bf16)
    yield model, cfg
    mesh_lib.set_default_mesh(None)


def _ids(seed=0):
    g = torch.Generator().manual_seed(seed)
    return torch.randint(1, 1024, (B, T), generator=g).cuda(), torch.randint(1, 1024, (STEPS, B, 1), generator=g).cuda()


def _run(model, cfg, recorded, monkeypatch, change=None, at=4, more=None):
    """Logits of a prompt and of ``STEPS`` steps, ``change(model)`` before step ``at``; and the cache."""
    from omegalax_b200.text import api

    monkeypatch.setenv("OMEGALAX_B200_DECODE_GRAPH", "1" if recorded else "0")
    prompt, steps = _ids()
    cache = api.make_cache(cfg, B, T, STEPS, device="cuda")
    out = [api.decode(model, cache, prompt, 0, cfg)[0]]
    for i, ids in enumerate(steps if more is None else more):
        if i == at:
            assert (cache.decode_graph is not None and cache.decode_graph[1] is not None) == recorded
            undo = change(model) if change else None
        out.append(api.decode(model, cache, ids, 0, cfg)[0].clone())
    if undo is not None:
        undo()
    return out, cache


def _replace(module, name):
    old = getattr(module, name)
    setattr(module, name, torch.nn.Parameter(-old.detach()))
    return lambda: setattr(module, name, old)


def _scalar(owner, name, value):
    old = getattr(owner, name)
    setattr(owner, name, value)
    return lambda: setattr(owner, name, old)


def _in_place(p):
    with torch.no_grad():
        p.neg_()
    return lambda: p.data.neg_()


def _narrow(mlp):      # half of the feed-forward's width, at the same addresses
    up, down = mlp.gate_up_proj.weight, mlp.down_proj.weight
    mlp.gate_up_proj.weight = torch.nn.Parameter(up.detach()[:512])
    mlp.down_proj.weight = torch.nn.Parameter(down.detach()[:, :256])

    def undo():
        mlp.gate_up_proj.weight, mlp.down_proj.weight = up, down
    return undo


def _forward(module):
    module.forward = lambda x, *a, **k: 0.5 * type(module).forward(module, x, *a, **k)
    return lambda: module.__dict__.pop("forward")


def _theta(model):
    old = model.cfg
    model.cfg = dataclasses.replace(old, rope_theta=100.0)
    return lambda: setattr(model, "cfg", old)


def _library(model):
    mp = pytest.MonkeyPatch()
    mp.setenv("OMEGALAX_B200_OPS", "library")
    return mp.undo


CHANGES = {
    "replaced weight": lambda m: _replace(m.layers[1].attn.o_proj, "weight"),
    "weight changed in place": lambda m: _in_place(m.layers[0].attn.qkv_proj.weight),
    "other shape at the same address": lambda m: _narrow(m.layers[0].mlp),
    "softmax scale": lambda m: _scalar(m.layers[0].attn, "scale", 0.5),
    "norm eps": lambda m: _scalar(m.layers[1].post_norm, "eps", 0.3),
    "query and key norm eps": lambda m: _scalar(m.layers[1].attn, "eps", 0.3),
    "rope theta": _theta,
    "forward of one module": lambda m: _forward(m.layers[0].post_norm),
    "hook": lambda m: m.layers[1].mlp.register_forward_hook(lambda mod, a, y: 2 * y).remove,
    "library ops": _library,
}


@pytest.mark.parametrize("what", CHANGES)
def test_a_change_between_steps_is_seen(served, monkeypatch, what):
    model, cfg = served
    monkeypatch.setattr("omegalax_b200.models.decode_graph.other_threads", lambda: False)
    state = {k: v.clone() for k, v in model.state_dict().items()}
    got, _ = _run(model, cfg, True, monkeypatch, CHANGES[what])
    for k, v in model.state_dict().items():
        assert torch.equal(v, state[k])
    want, _ = _run(model, cfg, False, monkeypatch, CHANGES[what])
    for i, (a, b) in enumerate(zip(got, want)):
        assert torch.equal(a, b), f"call {i}"


def test_idle_sequences_and_two_caches(served, monkeypatch):
    """A step without a token for one sequence between recorded ones; two caches whose steps alternate."""
    from omegalax_b200.text import api

    model, cfg = served
    monkeypatch.setattr("omegalax_b200.models.decode_graph.other_threads", lambda: False)
    more = _ids()[1].clone()
    more[5, 1] = 0
    got, _ = _run(model, cfg, True, monkeypatch, more=more)
    want, _ = _run(model, cfg, False, monkeypatch, more=more)
    for i, (a, b) in enumerate(zip(got, want)):
        assert torch.equal(a, b), f"call {i}"
    monkeypatch.setenv("OMEGALAX_B200_DECODE_GRAPH", "1")
    caches, outs = [api.make_cache(cfg, B, T, STEPS, device="cuda") for _ in range(2)], [[], []]
    for s in range(2):
        outs[s].append(api.decode(model, caches[s], _ids()[0], 0, cfg)[0])
    for ids in more:
        for s in range(2):
            outs[s].append(api.decode(model, caches[s], ids, 0, cfg)[0])
    for s in range(2):
        assert caches[s].decode_graph[1] is not None
        for a, b in zip(outs[s], want):
            assert torch.equal(a, b)


def test_a_step_that_runs_ahead_of_its_ids_leaves_the_cache_as_it_was(served, monkeypatch):
    """Sequences without a token at steps that need new pages, a cache that is full, and one whose pages are all taken: logits, lengths,
    pages and free list as when every step waits for its ids."""
    from omegalax_b200.text import api

    model, cfg = served
    monkeypatch.setattr("omegalax_b200.models.decode_graph.other_threads", lambda: False)
    steps = torch.randint(1, 1024, (14, B, 1), generator=torch.Generator().manual_seed(1)).cuda()
    steps[4, 1] = steps[9, 0] = steps[10] = 0      # 20 + 4 tokens fill three pages of 8, 20 + 12 four
    seen = []
    for recorded in (True, False):
        monkeypatch.setenv("OMEGALAX_B200_DECODE_GRAPH", "1" if recorded else "0")
        cache = api.make_cache(cfg, B, T, 12, device="cuda", page_size=8, num_pages=B * 4)
        out = [api.decode(model, cache, _ids()[0], 0, cfg)[0]]
        for ids in steps:
            try:
                out.append(api.decode(model, cache, ids, 0, cfg)[0].clone())
            except RuntimeError as e:
                out.append(torch.tensor([len(str(e))]))
            out.append(torch.tensor(cache.allocator.free + cache.seq_lens_host + cache.blocks_held))
            out.append(cache.block_table_host.clone())
        seen.append(out)
    for i, (a, b) in enumerate(zip(*seen)):
        assert torch.equal(a.cpu(), b.cpu()), i


@pytest.mark.parametrize("free,times", [(1 << 20, 1), (1 << 34, 0)])
def test_free_memory_of_the_allocator_is_given_back_where_a_recording_may_need_it(served, monkeypatch, free, times):
    """While a step is recorded the allocator cannot empty itself: done before, where the device has little left (a stand-in says how much)."""
    model, cfg = served
    monkeypatch.setattr("omegalax_b200.models.decode_graph.other_threads", lambda: False)
    want, _ = _run(model, cfg, False, monkeypatch, change=lambda m: lambda: None)
    calls, empty = [], torch.cuda.empty_cache

    def emptied():
        calls.append(torch.cuda.is_current_stream_capturing())
        empty()

    monkeypatch.setattr(torch.cuda, "mem_get_info", lambda *a: (free, 1 << 37))
    monkeypatch.setattr(torch.cuda, "empty_cache", emptied)
    got, _ = _run(model, cfg, True, monkeypatch, change=lambda m: lambda: None)
    assert calls == [False] * times
    for i, (a, b) in enumerate(zip(got, want)):
        assert torch.equal(a, b), f"call {i}"


def test_steps_on_two_streams(served, monkeypatch):
    """Steps of one cache that take turns on two streams: each finds lengths, pages and recorded buffers as the last one left them."""
    from omegalax_b200.text import api

    model, cfg = served
    monkeypatch.setattr("omegalax_b200.models.decode_graph.other_threads", lambda: False)
    want, _ = _run(model, cfg, False, monkeypatch)
    monkeypatch.setenv("OMEGALAX_B200_DECODE_GRAPH", "1")
    prompt, steps = _ids()
    cache = api.make_cache(cfg, B, T, STEPS, device="cuda")
    torch.cuda.synchronize()
    streams, out = [torch.cuda.Stream() for _ in range(2)], []
    for i, ids in enumerate([prompt, *steps]):
        with torch.cuda.stream(streams[i % 2]):
            out.append(api.decode(model, cache, ids, 0, cfg)[0])
            torch.empty(1 << 26, device="cuda").normal_()      # the next step, on the other stream, is issued long before this ends
    torch.cuda.synchronize()
    assert cache.decode_graph[1] is not None and cache.seq_lens.tolist() == [T + STEPS] * B
    for i, (a, b) in enumerate(zip(out, want)):
        assert torch.equal(a, b), f"call {i}"


def test_rows_of_pages_reserved_on_another_stream(served):
    """``flat_rows`` on one stream sees the pages whose table is still on its way on another."""
    from omegalax_b200.text import api

    cache = api.make_cache(served[1], B, 200, 0, device="cuda")
    seq = torch.arange(B, device="cuda").repeat_interleave(200)
    slot = torch.arange(200, device="cuda").repeat(B)
    work = torch.empty(1 << 28, device="cuda")
    torch.cuda.synchronize()
    with torch.cuda.stream(torch.cuda.Stream()):
        for _ in range(10):
            work.normal_()
        cache.reserve([200] * B)
    with torch.cuda.stream(torch.cuda.Stream()):
        rows = cache.flat_rows(seq, slot)
    torch.cuda.synchronize()
    assert rows.tolist() == [r for b in range(B) for r in cache.flat_rows_host(b, 0, 200).tolist()]


def test_nothing_is_recorded_beside_other_threads(served, monkeypatch):
    """Two threads that decode, draw random numbers and wait for the device at the same time: as when every call is issued."""
    import threading

    from omegalax_b200.text import api

    model, cfg = served
    want, _ = _run(model, cfg, False, monkeypatch)
    monkeypatch.setenv("OMEGALAX_B200_DECODE_GRAPH", "1")
    got, errors, start = [[], []], [], threading.Barrier(2)

    def serve(t):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                prompt, steps = _ids()
                cache = api.make_cache(cfg, B, T, STEPS, device="cuda")
                start.wait(30)
                for ids in [prompt, *steps]:
                    got[t].append(api.decode(model, cache, ids, 0, cfg)[0])
                    torch.multinomial(torch.softmax(got[t][-1].float(), -1), 1)
                    torch.cuda.synchronize()
                assert cache.decode_graph is None or cache.decode_graph[1] is None
        except BaseException as e:
            errors.append(e)

    torch.cuda.synchronize()
    threads = [threading.Thread(target=serve, args=(t,)) for t in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join(120)
    assert not errors and not any(t.is_alive() for t in threads)
    torch.cuda.synchronize()
    for t in range(2):
        for i, (a, b) in enumerate(zip(got[t], want)):
            assert torch.equal(a, b), f"thread {t} call {i}"
