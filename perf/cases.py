"""The measured work: fine-tuning steps and serving calls, through the entry points that the scripts use.

A case is one of three things:

* ``train``: one SFT step of ``trainers.text`` / ``trainers.vlm`` (copy of the batch from pinned memory, forward, loss,
  backward, clip, AdamW) on one GPU.  It gives loss, gradient norm and every parameter's first moment, which after the
  first step is the clipped gradient times 0.1.
* ``prompt``: ``text.api.decode`` of whole prompts into an empty paged cache: logits of every sequence's last token, and
  the cache.
* ``step``: ``text.api.decode`` of one more token for every sequence of a batch that has ``tokens`` cached.

Models have the widths of the presets and of ``bench.py`` and fewer layers.  All weights, ids and pixels are random;
norm weights are spread around one as trained ones are.
"""
import dataclasses
import math

import torch
import torch.nn.functional as F

BF16, F64 = torch.bfloat16, torch.float64
MORE = 256              # tokens a sequence of a ``step`` case may grow by before another takes its place

# preset, sizes of the layers, and how much of the model runs (layers of a training step, of a serving call)
QWEN = {
    "qwen3-0.6b": dict(id="Qwen/Qwen3-0.6B", V=151936, D=1024, F=3072, H=16, G=8, theta=1e6, train=4),
    "qwen3-8b": dict(id="Qwen/Qwen3-8B", V=151936, D=4096, F=12288, H=32, G=8, theta=1e6, train=2, serve=8),
    "qwen3-30b-a3b": dict(id="Qwen/Qwen3-30B-A3B-Instruct-2507", V=151936, D=2048, H=32, G=4, theta=1e7, E=128, top=8, FE=768,
                          train=2),
    "qwen3-vl-2b": dict(id="Qwen/Qwen3-VL-2B-Instruct", V=151936, D=2048, F=6144, H=16, G=8, theta=5e6, train=2),
}
HYBRID = dict(id="qwen3.5-397b-a17b-8layer", V=32768, D=4096, H=32, G=2, E=32, top=10, FE=1024, train=2)     # one layer of each kind
LETITAR = dict(id="letitar-8layer-4096", V=151936, D=4096, F=18432, serve=8)
DIFEDRA = dict(id="difedra-8layer-2048", V=151936, D=2048, H=32, G=4, E=128, top=8, FE=768, F=6144, serve=8)
VIT = dict(D=1024, F=4096, H=16, depth=2, out=2048, side=48)
SERVED = ("qwen3-8b", "letitar", "difedra")
ROUTED = ("qwen3-30b-a3b", "qwen3.5", "difedra")


def listed():
    train, prompt, step = dict(do="train"), dict(do="prompt"), dict(do="step")
    return [
        # the headline fine-tuning work: long packed rows of the 8B width
        dict(train, name="train 8b 2x4096", model="qwen3-8b", batch=2, tokens=4096, ragged=False),
        # a small model on short padded conversations: latency and launches count
        dict(train, name="train 0.6b 3x333 padded", model="qwen3-0.6b", batch=3, tokens=333, ragged=True),
        # routed experts, whole rows
        dict(train, name="train 30b-a3b 1x4096", model="qwen3-30b-a3b", batch=1, tokens=4096, ragged=False),
        # hybrid of gated delta rule and gated attention, a row that no tile divides
        dict(train, name="train qwen3.5 1x3001", model="qwen3.5", batch=1, tokens=3001, ragged=False),
        # images with text: one 448 x 448 image and a conversation per row
        dict(train, name="train vl 4x1220", model="qwen3-vl-2b", batch=4, tokens=1220, ragged=False, grid_h=28, grid_w=28),
        # one long document read at once, and a batch of prompts of mixed lengths
        dict(prompt, name="prompt 8b 1x8192", model="qwen3-8b", batch=1, tokens=8192, ragged=False),
        dict(prompt, name="prompt letitar 8x1024 mixed", model="letitar", batch=8, tokens=1024, ragged=True),
        # a chat turn
        dict(prompt, name="prompt difedra 1x500", model="difedra", batch=1, tokens=500, ragged=False),
        # one user, long context; a batch of users; many users with short contexts
        dict(step, name="step 8b 1x4096", model="qwen3-8b", batch=1, tokens=4096, ragged=False),
        dict(step, name="step 8b 32x2048", model="qwen3-8b", batch=32, tokens=2048, ragged=False),
        dict(step, name="step letitar 16x2048", model="letitar", batch=16, tokens=2048, ragged=False),
        dict(step, name="step difedra 64x1000", model="difedra", batch=64, tokens=1000, ragged=False),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    do = rng.choice(("train", "prompt", "step"))
    if do == "train":
        model = rng.choice((*QWEN, "qwen3.5"))
        batch = rng.randint(1, 4)
        if model == "qwen3-vl-2b":
            gh, gw = 2 * rng.randint(4, 14), 2 * rng.randint(4, 14)
            return dict(do=do, model=model, batch=batch, tokens=gh * gw // 4 + 1 + _log(rng, 32, 1024), ragged=False, grid_h=gh, grid_w=gw)
        most = 4096 if model in ("qwen3-30b-a3b", "qwen3.5") else 8192
        return dict(do=do, model=model, batch=batch, tokens=_log(rng, 48, min(4096, most // batch)),
                    ragged=model in ("qwen3-0.6b", "qwen3-8b") and rng.random() < 0.5)
    model = rng.choice(SERVED)
    if do == "prompt":
        batch = rng.randint(1, 8)
        return dict(do=do, model=model, batch=batch, tokens=_log(rng, 16, 8192 // batch), ragged=rng.random() < 0.5)
    batch = _log(rng, 1, 128)
    return dict(do=do, model=model, batch=batch, tokens=_log(rng, 16, min(4096, 65536 // batch)), ragged=rng.random() < 0.5)


def _lengths(case):
    """Tokens of every row: all of them, or down to half of them."""
    B, T = case["batch"], case["tokens"]
    return [T - (b * 2654435761 % 1000) * (T // 2) // 1000 if case["ragged"] else T for b in range(B)]


# ------------------------------------------------------------------------------------------------ inputs
def _qwen_layer(p, m):
    q, kv, D = m["H"] * 128, m["G"] * 128, m["D"]
    out = [(p + "input_norm.weight", (D,)), (p + "attn.qkv_proj.weight", (q + 2 * kv, D)), (p + "attn.o_proj.weight", (D, q)),
           (p + "attn.q_norm.weight", (128,)), (p + "attn.k_norm.weight", (128,)), (p + "post_norm.weight", (D,))]
    if "E" in m:
        return out + [(p + "mlp.router.weight", (m["E"], D)), (p + "mlp.experts_gate_up", (m["E"], 2 * m["FE"], D)),
                      (p + "mlp.experts_down", (m["E"], D, m["FE"]))]
    return out + [(p + "mlp.gate_up_proj.weight", (2 * m["F"], D)), (p + "mlp.down_proj.weight", (D, m["F"]))]


def _hybrid_layer(p, m, linear):
    D, E, FE = m["D"], m["E"], m["FE"]
    out = [(p + "input_norm.weight", (D,)), (p + "post_norm.weight", (D,))]
    if linear:
        a = p + "linear_attn."
        out += [(a + "in_proj_qkv.weight", (12288, D)), (a + "in_proj_z.weight", (8192, D)), (a + "in_proj_b.weight", (64, D)),
                (a + "in_proj_a.weight", (64, D)), (a + "conv_weight", (12288, 4)), (a + "dt_bias", (64,)), (a + "A_log", (64,)),
                (a + "norm.weight", (128,)), (a + "out_proj.weight", (D, 8192))]
    else:
        a = p + "attn."
        out += [(a + "qkv_proj.weight", ((2 * m["H"] + 2 * m["G"]) * 256, D)), (a + "o_proj.weight", (D, m["H"] * 256)),
                (a + "q_norm.weight", (256,)), (a + "k_norm.weight", (256,))]
    return out + [(p + "mlp.router.weight", (E, D)), (p + "mlp.experts_gate_up", (E, 2 * FE, D)), (p + "mlp.experts_down", (E, D, FE)),
                  (p + "mlp.shared_expert.gate_up_proj.weight", (2 * FE, D)), (p + "mlp.shared_expert.down_proj.weight", (D, FE)),
                  (p + "mlp.shared_expert_gate.weight", (1, D))]


def _vision(p):
    D, Fv, G4 = VIT["D"], VIT["F"], 4 * VIT["D"]

    def dense(n, o, i):
        return [(n + ".weight", (o, i)), (n + ".bias", (o,))]

    def norm(n, d):
        return [(n + ".weight", (d,)), (n + ".bias", (d,))]

    out = [(p + "pos_embed", (VIT["side"] ** 2, D))] + dense(p + "patch_embed", D, 1536)
    for i in range(VIT["depth"]):
        b = f"{p}blocks.{i}."
        out += norm(b + "norm1", D) + norm(b + "norm2", D) + dense(b + "attn.qkv", 3 * D, D) + dense(b + "attn.proj", D, D)
        out += dense(b + "mlp.linear_fc1", Fv, D) + dense(b + "mlp.linear_fc2", D, Fv)
    for g, n in ((p + "merger.", D), (p + "deepstack_mergers.0.", G4)):
        out += norm(g + "norm", n) + dense(g + "linear_fc1", G4, G4) + dense(g + "linear_fc2", VIT["out"], G4)
    return out


def _shapes(case):
    """(name, shape) of every parameter."""
    name, n = case["model"], _layers(case)
    if name in QWEN:
        m = QWEN[name]
        out = _vision("visual.") if name == "qwen3-vl-2b" else []
        out += [("embedder.weight", (m["V"], m["D"]))]
        for i in range(n):
            out += _qwen_layer(f"layers.{i}.", m)
        return out + [("final_norm.weight", (m["D"],)), ("lm_head.weight", (m["V"], m["D"]))]
    if name == "qwen3.5":
        out = [("model.embedder.weight", (HYBRID["V"], HYBRID["D"]))]
        for i in range(n):
            out += _hybrid_layer(f"model.layers.{i}.", HYBRID, i % 2 == 0)
        return out + [("model.final_norm.weight", (HYBRID["D"],)), ("lm_head.weight", (HYBRID["V"], HYBRID["D"]))]
    m = LETITAR if name == "letitar" else DIFEDRA
    D = m["D"]
    out = [("embedder.weight", (m["V"], D))]
    for i in range(n):
        p = f"layers.{i}."
        out += [(p + "norm1.weight", (D,)), (p + "norm2.weight", (D,))]
        if name == "letitar":
            out += [(p + "norm1.bias", (D,)), (p + "norm2.bias", (D,)), (p + "mlp.up.weight", (m["F"], D)),
                    (p + "mlp.down.weight", (D, m["F"])), (p + "mixer.out_proj.weight", (D, 4096))]
            if i in (0, 4, 7):
                out += [(p + "mixer.in_proj.weight", (6144 + (576 if i < 7 else 0), D)), (p + "mixer.kv_proj.weight", (8192, 512))]
                out += [(p + "mixer.latent_norm", (512,))] if i < 7 else []
            else:
                out += [(p + "mixer.in_proj.weight", (4 * 4096 + 32, D)), (p + "mixer.decay_proj.weight", (4096, 32)),
                        (p + "mixer.decay_bias", (4096,)), (p + "mixer.norm_weight", (128,))]
        else:
            out += [(p + "mixer.in_proj.weight", (5120, D)), (p + "mixer.qk_norm", (4608,)), (p + "mixer.value_mix", ()),
                    (p + "mixer.sink", (32,)), (p + "mixer.out_proj.weight", (D, 4096))]
            if i == 0:
                out += [(p + "mlp.gate_up.weight", (2 * m["F"], D)), (p + "mlp.down.weight", (D, m["F"]))]
            else:
                out += [(p + "mlp.router.weight", (m["E"], D)), (p + "mlp.experts_gate_up", (m["E"], 2 * m["FE"], D)),
                        (p + "mlp.experts_down", (m["E"], D, m["FE"]))]
    out.append(("final_norm.weight", (D,)))
    return out + ([("final_norm.bias", (D,)), ("lm_head.weight", (m["V"], D))] if name == "letitar" else [])


def _spread(case, name, shape):
    """Mean and standard deviation of a parameter."""
    if name.endswith("A_log"):
        return 1.5, 0.8
    if name.endswith("dt_bias"):
        return 1.0, 0.5
    if name.endswith("value_mix"):
        return 0.4, 0.1
    if name.endswith("sink"):
        return 0.0, 1.0
    if name.endswith((".bias", "decay_bias")):
        return 0.0, 0.1
    if len(shape) == 1:
        one_plus = case["model"] == "qwen3.5" and not name.endswith("linear_attn.norm.weight")
        return (0.0 if one_plus else 1.0), 0.1
    if name.endswith(("embedder.weight", "pos_embed")):
        return 0.0, (1.0 if case["model"] in ROUTED or case["model"] == "letitar" else 0.02)
    if case["model"] in ROUTED and name.endswith(("o_proj.weight", "out_proj.weight", "down", "down.weight", "down_proj.weight")):
        return 0.0, 0.25 * shape[-1] ** -0.5        # a layer adds a fraction of what the residual rows hold
    return 0.0, shape[-1] ** -0.5


def _device():
    return torch.device("cuda", torch.cuda.current_device()) if torch.cuda.is_available() else torch.device("cpu")


def _weights(case, seed):
    """bf16 values of every parameter, by name."""
    dev = _device()
    g = torch.Generator(device=dev).manual_seed(seed * 7919 + 1)
    out = {}
    for name, shape in _shapes(case):
        mean, std = _spread(case, name, shape)
        out[name] = torch.randn(shape, generator=g, device=dev, dtype=BF16).mul_(std).add_(mean)
    if case["model"] in ROUTED:
        _specialise(case, out, g)
    return out


def _specialise(case, w, g):
    """Routers as training leaves them: a token has experts of its own in every layer, ahead of the others by a margin.  (With
    independent random routers a twentieth of the tokens would change experts with the last bit of any sum.)"""
    table = next(v for k, v in w.items() if k.endswith("embedder.weight"))
    routers = [v for k, v in w.items() if k.endswith("router.weight")]
    (E, D), top = routers[0].shape, 10 if case["model"] == "qwen3.5" else 8
    rows = routers[0].clone()
    for i, r in enumerate(routers):
        r.copy_(rows[torch.randperm(E, generator=g, device=g.device)] if i else rows).mul_(0.4)
    for part in table.split(16384):
        own = torch.rand(part.shape[0], E, generator=g, device=g.device).topk(top, -1).indices
        hot = torch.zeros(part.shape[0], E, dtype=BF16, device=g.device).scatter_(1, own, 1.0)
        part.add_(hot @ rows, alpha=0.5 * (D / top) ** 0.5)


def _vocab(case):
    name = case["model"]
    return (QWEN[name] if name in QWEN else HYBRID if name == "qwen3.5" else LETITAR if name == "letitar" else DIFEDRA)["V"]


def _layers(case):
    name = case["model"]
    m = QWEN[name] if name in QWEN else HYBRID if name == "qwen3.5" else LETITAR if name == "letitar" else DIFEDRA
    return m["train" if case["do"] == "train" else "serve"]


def _rows(case, seed):
    """Token ids [batch, tokens + 1 for a step] on the host, 0 where a row has ended, and rows of ids for the steps."""
    g = torch.Generator().manual_seed(seed * 7919 + 2)
    B, T, V = case["batch"], case["tokens"], min(_vocab(case), 151643)      # ids above are control tokens
    ids = torch.randint(1, V, (B, T), generator=g, dtype=torch.int32)
    for b, n in enumerate(_lengths(case)):
        ids[b, n:] = 0
    return ids, torch.randint(1, V, (MORE, B, 1), generator=g, dtype=torch.int32)


def _batch(case, seed):
    """The batch of a training step in pinned memory, as the collators lay it out: the second half is supervised."""
    ids, _ = _rows(case, seed)
    B, T = ids.shape
    real = (ids != 0).to(torch.int32)
    loss = real.clone()
    loss[:, : T // 2] = 0
    out = {"token_ids_BT": ids, "attention_mask_BT": real, "loss_mask_BT": loss}
    if case["model"] == "qwen3-vl-2b":
        gh, gw = case["grid_h"], case["grid_w"]
        n = gh * gw // 4
        ids[:, 0], ids[:, 1:1 + n] = 151652, 151655
        g = torch.Generator().manual_seed(seed * 7919 + 3)
        out["pixel_values"] = torch.randn(B * gh * gw, 1536, generator=g)
        out["image_grid_thw"] = torch.tensor([[1, gh, gw]] * B, dtype=torch.int32)
        out["vision_cu_seqlens"] = torch.arange(B + 1, dtype=torch.int32) * (gh * gw)
        pos = torch.zeros(3, T, dtype=torch.int32)
        pos[0, 1:1 + n] = 1
        pos[1, 1:1 + n] = 1 + torch.arange(gh // 2, dtype=torch.int32).repeat_interleave(gw // 2)
        pos[2, 1:1 + n] = 1 + torch.arange(gw // 2, dtype=torch.int32).repeat(gh // 2)
        pos[:, 1 + n:] = 1 + max(gh, gw) // 2 + torch.arange(T - 1 - n, dtype=torch.int32)
        out["position_ids_ZBT"] = pos[:, None].expand(3, B, T).contiguous()
    return {k: v.pin_memory() if torch.cuda.is_available() else v for k, v in out.items()}


# ------------------------------------------------------------------------------------------------ the program
def _model(case, seed):
    from omegalax_b200.text import api as text_api
    from omegalax_b200.vlm import api as vlm_api

    name, n = case["model"], _layers(case)
    api = vlm_api if name == "qwen3-vl-2b" else text_api
    if name == "qwen3.5":
        cfg = dataclasses.replace(api.resolve_config(HYBRID["id"]), num_hidden_layers=n, num_experts=HYBRID["E"], vocab_size=HYBRID["V"],
                                  layer_types=("linear_attention", "full_attention") * (n // 2))
    elif name in QWEN:
        cfg = dataclasses.replace(api.resolve_config(QWEN[name]["id"]), num_layers=n)
        if name == "qwen3-vl-2b":
            cfg = dataclasses.replace(cfg, vision=dataclasses.replace(cfg.vision, depth=VIT["depth"], deepstack_visual_indexes=(0,)))
    else:
        cfg = api.resolve_config((LETITAR if name == "letitar" else DIFEDRA)["id"])
    model, cfg = api.init_model(cfg, 0, tp_size=1, fsdp_size=1, dp_size=1, device=_device(), dtype=BF16)
    w = _weights(case, seed)
    with torch.no_grad():
        for key, p in model.named_parameters():
            p.copy_(w.pop(key))
    if w:
        raise RuntimeError(f"parameters that the model does not have: {sorted(w)}")
    return model, cfg, api


def prepare(case, seed):
    from omegalax_b200.trainers import text as text_trainer
    from omegalax_b200.trainers import vlm as vlm_trainer

    model, cfg, api = _model(case, seed)
    if case["do"] == "train":
        trainer = vlm_trainer if case["model"] == "qwen3-vl-2b" else text_trainer
        tcfg = trainer.TrainConfig(batch_size=case["batch"], seq_len=case["tokens"], num_steps=10_000, learning_rate=1e-5,
                                   max_grad_norm=1.0, remat_policy="full" if case["model"] == "qwen3.5" else "selective")
        opt = trainer.build_optimizer(model, tcfg, device=_device())
        names = {id(p): n for n, p in model.named_parameters()}
        moments = {names[id(s.param)]: m.view(s.shape) for s, _, m, _ in opt.named_master_shards()}
        return {"case": case, "api": api, "cfg": cfg, "opt": opt, "batch": _batch(case, seed), "moments": moments,
                "step": trainer.make_sft_train_step(cfg, pad_id=0)}
    B, T, n = case["batch"], case["tokens"], _lengths(case)
    ids, more = _rows(case, seed)
    if case["model"] == "qwen3-8b":          # this family takes its ids on the device
        ids, more = ids.to(_device()), more.to(_device())
    cache = api.make_cache(cfg, B, T, 0 if case["do"] == "prompt" else MORE, device=_device())
    state = {"case": case, "api": api, "cfg": cfg, "model": model, "cache": cache, "ids": ids, "more": more, "lengths": n, "used": 0}
    if case["do"] == "step":
        _, state["cache"], _ = api.decode(model, cache, ids, 0, cfg)
    return state


def run(state):
    case, api, cfg = state["case"], state["api"], state["cfg"]
    if case["do"] == "train":
        batch = api.shard_batch_dict(state["batch"], cfg, device=_device())
        loss, metrics = state["step"](state["opt"], batch)
        return {"loss": loss, "grad_norm": metrics["grad_norm"], "moments": state["moments"]}
    cache, B = state["cache"], case["batch"]
    if case["do"] == "prompt":
        for b in range(B):
            cache.free_sequence(b)
        logits, _, _ = api.decode(state["model"], cache, state["ids"], 0, cfg)
        return {"logits": logits, "cache": _stores(cache)}
    if state["used"] == MORE:               # the sequences end, and others with as many tokens take their places
        for b in range(B):
            cache.free_sequence(b)
        cache.reserve(state["lengths"])
        cache.advance(state["lengths"])
        state["used"] = 0
    logits, _, _ = api.decode(state["model"], cache, state["more"][state["used"]], 0, cfg)
    state["used"] += 1
    return {"logits": logits, "cache": _stores(cache)}


def _stores(cache):
    """What the layers keep: pages of keys and values or latents, recurrent states."""
    return cache.stores if hasattr(cache, "stores") else cache.k_pages + cache.v_pages


# ------------------------------------------------------------------------------------------------ what it costs
def _active(case, tokens):
    """(parameters that ``tokens`` tokens read at least once, multiply-adds of one token in products with weights), without
    the embedding table and the head."""
    name, read, macs = case["model"], 0.0, 0.0
    for key, shape in _shapes(case):
        k = math.prod(shape)
        if key.startswith("visual.") or key.endswith(("embedder.weight", "lm_head.weight")):
            continue
        if ".experts_" in key:
            E, top = shape[0], 10 if name == "qwen3.5" else 8
            read += k * (1 - (1 - top / E) ** tokens)
            macs += k / E * top
        else:
            read += k
            macs += k
    return read, macs


def work(case):
    n, B = _lengths(case), case["batch"]
    V, name = _vocab(case), case["model"]
    D = (QWEN[name] if name in QWEN else HYBRID if name == "qwen3.5" else LETITAR if name == "letitar" else DIFEDRA)["D"]
    # channels of queries and keys, and of values, over all heads of all attention layers; recurrent heads x state entries
    attn = {"letitar": 3 * 32 * (192 + 128), "difedra": 8 * 32 * 256, "qwen3.5": 32 * 512}.get(name) or _layers(case) * QWEN[name]["H"] * 256
    state = {"letitar": 5 * 32 * 128 * 128, "qwen3.5": 64 * 128 * 128}.get(name, 0)
    cached = {"letitar": 2 * 576, "difedra": 8 * 4 * 256}.get(name) or (0 if name == "qwen3.5" else _layers(case) * QWEN[name]["G"] * 256)
    if case["do"] == "train":
        M = sum(n)
        total = sum(math.prod(s) for _, s in _shapes(case))
        flops = 6.0 * M * (_active(case, M)[1] + V * D) + 3.5 * attn * sum(t * t for t in n) + 3 * 6.0 * state * M
        if name == "qwen3-vl-2b":
            P = case["grid_h"] * case["grid_w"]
            flops += 6.0 * B * P * sum(math.prod(s) * (0.25 if "merger" in k else 1) for k, s in _vision("") if len(s) == 2)
            flops += 3.5 * VIT["depth"] * 2 * VIT["D"] * 2 * B * P * P
        # weights, two moments and the 16-bit copy, each read and written
        return {"bytes": 28.0 * total, "flops": flops}
    if case["do"] == "prompt":
        M = sum(n)
        read, macs = _active(case, M)
        return {"bytes": 2.0 * (read + V * D + M * cached) + 4.0 * B * (V + state),
                "flops": 2.0 * (M * macs + B * V * D) + attn * sum(t * t for t in n) + 6.0 * state * M}
    read, macs = _active(case, B)
    keys = sum(n) + B
    return {"bytes": 2.0 * (read + V * D + keys * cached) + 4.0 * B * (V + 2 * state),
            "flops": 2.0 * B * (macs + V * D) + 2.0 * attn * keys + 6.0 * state * B}


def tolerance(case):
    # Activations and gradients between kernels are bf16.  Against 64 bits, logits are off by 0.014 (8 Qwen3 layers), 0.0095
    # (Letitar) and 0.004 (Difedra), moments by up to 0.02, and two correct sums in different orders differ by as much
    # (Letitar's projections with and without a split reduction: rel 0.0085, max 0.056; embedding gradients of one and the
    # same program with sums by atomics: rel 0.002, max 0.048).
    return {"rel": 0.03, "max": 0.6}


# ------------------------------------------------------------------------------------------------ the same in 64 bits
def _rms(x, w, eps=1e-6):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * w


def _turn(x, ang, rot):
    """Channels i and i + rot/2 of x [N, heads, K] turned by ang [N, rot/2]."""
    c, s = ang.cos()[:, None], ang.sin()[:, None]
    a, b = x[..., : rot // 2], x[..., rot // 2: rot]
    return torch.cat([a * c - b * s, b * c + a * s, x[..., rot:]], -1)


def _turn_pairs(x, ang, amp):
    c, s = ang.cos()[:, None] * amp, ang.sin()[:, None] * amp
    a, b = x[..., 0::2], x[..., 1::2]
    return torch.stack([a * c - b * s, b * c + a * s], -1).flatten(-2)


def _attend(q, k, v, lengths, scale, causal=True, sink=None):
    """q [N, H, K], k and v [N, G, *] of packed sequences.  A few heads at a time, which bounds the scores."""
    out, at, rep = [], 0, q.shape[1] // k.shape[1]
    for n in lengths:
        i = slice(at, at + n)
        hidden = torch.ones(n, n, dtype=torch.bool, device=q.device).triu(1) if causal else None
        heads, per = [], max(1, (1 << 28) // (n * n))
        for h in range(0, q.shape[1], per):
            hs = torch.arange(h, min(h + per, q.shape[1]), device=q.device)
            s = q[i, hs].transpose(0, 1) @ k[i, hs // rep].permute(1, 2, 0) * scale
            if hidden is not None:
                s = s.masked_fill(hidden, -math.inf)
            if sink is not None:
                s = torch.cat([s, sink[hs][:, None, None].expand(-1, n, 1)], -1)
            p = torch.softmax(s, -1)[..., :n]
            heads.append((p @ v[i, hs // rep].transpose(0, 1)).transpose(0, 1))
        out.append(torch.cat(heads, 1))
        at += n
    return torch.cat(out)


def _experts(h, weight, idx, gate_up, down, on_input):
    out = torch.zeros_like(h)
    for e in range(gate_up.shape[0]):
        tok, slot = (idx == e).nonzero(as_tuple=True)
        if not tok.numel():
            continue
        a = weight[tok, slot][:, None]
        g, u = ((h[tok] * a if on_input else h[tok]) @ gate_up[e].to(F64).t()).chunk(2, -1)
        y = (F.silu(g) * u) @ down[e].to(F64).t()
        out = out.index_add(0, tok, y if on_input else y * a)
    return out


def _qwen_forward(w, m, x, ang, lengths, n, deep=None):
    """Packed rows x after the layers, and the load-balance loss."""
    aux = x.new_zeros(())
    for i in range(n):
        p = f"layers.{i}."
        W = lambda key: w[p + key].to(F64)  # noqa: E731
        N, H, G = x.shape[0], m["H"], m["G"]
        q, k, v = (_rms(x, W("input_norm.weight")) @ W("attn.qkv_proj.weight").t()).view(N, -1, 128).split([H, G, G], 1)
        q = _turn(_rms(q, W("attn.q_norm.weight")), ang, 128)
        k = _turn(_rms(k, W("attn.k_norm.weight")), ang, 128)
        x = x + _attend(q, k, v, lengths, 128 ** -0.5).reshape(N, -1) @ W("attn.o_proj.weight").t()
        h = _rms(x, W("post_norm.weight"))
        if "E" in m:
            probs = torch.softmax(h @ W("mlp.router.weight").t(), -1)
            top, idx = probs.topk(m["top"], -1)
            x = x + _experts(h, top / top.sum(-1, keepdim=True), idx, w[p + "mlp.experts_gate_up"], w[p + "mlp.experts_down"], False)
            count = torch.bincount(idx.reshape(-1), minlength=m["E"]).to(F64)
            aux = aux + 0.001 * m["E"] * (count / N * probs.mean(0)).sum()
        else:
            up, down = W("mlp.gate_up_proj.weight"), W("mlp.down_proj.weight")
            parts = []
            for c in h.split(16384):
                g, u = (c @ up.t()).chunk(2, -1)
                parts.append((F.silu(g) * u) @ down.t())
            x = x + torch.cat(parts)
        if deep is not None and i == 0:
            x = x.index_add(0, deep[0], deep[1])
    return x, aux


def _delta_rule(q, k, v, g, beta):
    """Gated delta rule over one sequence: q, k [T, H, A], v [T, H, U], g and beta [T, H]; chunks of 64."""
    T, C = q.shape[0], 64
    pad = -T % C
    q, k, v = (F.pad(t, (0, 0, 0, 0, 0, pad)).unflatten(0, (-1, C)).transpose(1, 2) for t in (q, k, v))      # [J, H, C, *]
    g, beta = (F.pad(t, (0, 0, 0, pad)).unflatten(0, (-1, C)).transpose(1, 2) for t in (g, beta))
    G = g.cumsum(-1)
    low = torch.ones(C, C, dtype=torch.bool, device=q.device).tril()
    decay = torch.exp((G[..., :, None] - G[..., None, :]).masked_fill(~low, -math.inf))
    kk = (k @ k.transpose(-1, -2)) * decay * beta[..., None]
    eye = torch.eye(C, dtype=F64, device=q.device)
    rhs = torch.cat([v * beta[..., None], k * (beta * torch.exp(G))[..., None]], -1)
    solved = torch.linalg.solve_triangular(kk.tril(-1) + eye, rhs, upper=False, unitriangular=True)
    u, z = solved[..., : v.shape[-1]], solved[..., v.shape[-1]:]
    inner = (q @ k.transpose(-1, -2)) * decay
    S, out = q.new_zeros(q.shape[1], q.shape[-1], v.shape[-1]), []
    for j in range(q.shape[0]):
        fresh = u[j] - z[j] @ S
        out.append((q[j] * torch.exp(G[j])[..., None]) @ S + inner[j] @ fresh)
        last = G[j, :, -1:]
        S = S * torch.exp(last)[..., None] + (k[j] * torch.exp(last - G[j])[..., None]).transpose(-1, -2) @ fresh
    return torch.stack(out).transpose(1, 2).flatten(0, 1)[:T]


def _hybrid_forward(w, x, lengths, n):
    T, B, m, aux = lengths[0], len(lengths), HYBRID, x.new_zeros(())
    pos = torch.arange(T, dtype=F64, device=x.device).repeat(B)
    ang = pos[:, None] * 1e7 ** (-torch.arange(0, 64, 2, dtype=F64, device=x.device) / 64)
    for i in range(n):
        p = f"model.layers.{i}."
        W = lambda key: w[p + key].to(F64)  # noqa: E731
        N, h = x.shape[0], _rms(x, 1 + W("input_norm.weight"))
        if i % 2 == 0:
            a = "linear_attn."
            mixed, z = (h @ W(a + "in_proj_qkv.weight").t()).view(B, T, -1), h @ W(a + "in_proj_z.weight").t()
            beta = torch.sigmoid(h @ W(a + "in_proj_b.weight").t())
            g = -torch.exp(W(a + "A_log")) * F.softplus(h @ W(a + "in_proj_a.weight").t() + W(a + "dt_bias"))
            past, kern = F.pad(mixed, (0, 0, 3, 0)), W(a + "conv_weight")
            mixed = F.silu(sum(past[:, t: t + T] * kern[:, t] for t in range(4))).reshape(N, -1)
            q, k, v = (t.view(N, -1, 128) for t in mixed.split([2048, 2048, 8192], -1))
            q, k = (t * torch.rsqrt(t.square().sum(-1, keepdim=True) + 1e-6) for t in (q, k))
            q, k = (t.repeat_interleave(4, 1) for t in (q * 128 ** -0.5, k))
            o = torch.cat([_delta_rule(*(t[b * T: (b + 1) * T] for t in (q, k, v, g, beta))) for b in range(B)])
            o = _rms(o, W(a + "norm.weight")) * F.silu(z.view(N, -1, 128))
            x = x + o.reshape(N, -1) @ W(a + "out_proj.weight").t()
        else:
            qkv = (h @ W("attn.qkv_proj.weight").t()).view(N, -1, 256)
            q, k, v = qkv.split([2 * m["H"], m["G"], m["G"]], 1)
            q, gate = q[:, 0::2], q[:, 1::2]
            q, k = _turn(_rms(q, 1 + W("attn.q_norm.weight")), ang, 64), _turn(_rms(k, 1 + W("attn.k_norm.weight")), ang, 64)
            o = _attend(q, k, v, lengths, 256 ** -0.5) * torch.sigmoid(gate)
            x = x + o.reshape(N, -1) @ W("attn.o_proj.weight").t()
        h = _rms(x, 1 + W("post_norm.weight"))
        probs = torch.softmax(h @ W("mlp.router.weight").t(), -1)
        top, idx = probs.topk(m["top"], -1)
        y = _experts(h, top / top.sum(-1, keepdim=True), idx, w[p + "mlp.experts_gate_up"], w[p + "mlp.experts_down"], False)
        g, u = (h @ W("mlp.shared_expert.gate_up_proj.weight").t()).chunk(2, -1)
        y = y + torch.sigmoid(h @ W("mlp.shared_expert_gate.weight").t()) * ((F.silu(g) * u) @ W("mlp.shared_expert.down_proj.weight").t())
        x = x + y
        aux = aux + 0.001 * ((probs.mean(0) - 1 / m["E"]) ** 2).sum()
    return x, aux


def _vision_forward(w, pixels, gh, gw, B):
    """Image features, and the tapped ones that the first decoder layer adds."""
    W = lambda key: w["visual." + key].to(F64)  # noqa: E731
    dev, D, H, side = pixels.device, VIT["D"], VIT["H"], VIT["side"]
    dense = lambda x, n: x @ W(n + ".weight").t() + W(n + ".bias")  # noqa: E731
    norm = lambda x, n: F.layer_norm(x, x.shape[-1:], W(n + ".weight"), W(n + ".bias"), 1e-6)  # noqa: E731
    row = torch.arange(gh, device=dev)[:, None].expand(gh, gw)
    col = torch.arange(gw, device=dev)[None, :].expand(gh, gw)
    order = lambda t: t.reshape(gh // 2, 2, gw // 2, 2, *t.shape[2:]).transpose(1, 2).flatten(0, 3)  # noqa: E731  2 x 2 blocks together
    hi, wi = (torch.linspace(0, side - 1, s, device=dev).to(F64) for s in (gh, gw))
    h0, w0 = hi.floor().long(), wi.floor().long()
    h1, w1 = (h0 + 1).clamp(max=side - 1), (w0 + 1).clamp(max=side - 1)
    dh, dw = (hi - h0)[:, None, None], (wi - w0)[None, :, None]
    at = lambda a, b: W("pos_embed")[a[:, None] * side + b[None, :]]  # noqa: E731
    pe = (1 - dh) * ((1 - dw) * at(h0, w0) + dw * at(h0, w1)) + dh * ((1 - dw) * at(h1, w0) + dw * at(h1, w1))
    x = dense(pixels.to(F64), "patch_embed") + order(pe).repeat(B, 1)
    inv = 10000.0 ** (-torch.arange(0, 32, 2, dtype=F64, device=dev) / 32)
    ang = torch.cat([order(row)[:, None] * inv, order(col)[:, None] * inv], -1).repeat(B, 1)
    tapped = None
    for i in range(VIT["depth"]):
        b = f"blocks.{i}."
        q, k, v = dense(norm(x, b + "norm1"), b + "attn.qkv").view(-1, 3, H, D // H).unbind(1)
        o = _attend(_turn(q, ang, D // H), _turn(k, ang, D // H), v, [gh * gw] * B, (D // H) ** -0.5, causal=False)
        x = x + dense(o.reshape(-1, D), b + "attn.proj")
        x = x + dense(F.gelu(dense(norm(x, b + "norm2"), b + "mlp.linear_fc1"), approximate="tanh"), b + "mlp.linear_fc2")
        if i == 0:
            t = norm(x.view(-1, 4 * D), "deepstack_mergers.0.norm")
            tapped = dense(F.gelu(dense(t, "deepstack_mergers.0.linear_fc1")), "deepstack_mergers.0.linear_fc2")
    t = norm(x, "merger.norm").view(-1, 4 * D)
    return dense(F.gelu(dense(t, "merger.linear_fc1")), "merger.linear_fc2"), tapped


def _exact_train(case, seed):
    dev, name, n = _device(), case["model"], _layers(case)
    w = {k: v.to(F64).requires_grad_() for k, v in _weights(case, seed).items()}
    batch = {k: v.to(dev) for k, v in _batch(case, seed).items()}
    ids = batch["token_ids_BT"].long()
    B, T = ids.shape
    pre = "model." if name == "qwen3.5" else ""
    x = w[pre + "embedder.weight"][ids.reshape(-1)]
    if name == "qwen3.5":
        x, aux = _hybrid_forward(w, x, [T] * B, n)
        x = _rms(x, 1 + w[pre + "final_norm.weight"])
    else:
        m, deep = QWEN[name], None
        inv = m["theta"] ** (-torch.arange(0, 128, 2, dtype=F64, device=dev) / 128)
        if name == "qwen3-vl-2b":
            feats, tapped = _vision_forward(w, batch["pixel_values"].to(BF16), case["grid_h"], case["grid_w"], B)
            where = (ids.reshape(-1) == 151655).nonzero().squeeze(1)
            x = x.index_copy(0, where, feats)
            deep = (where, tapped)
            f = batch["position_ids_ZBT"].to(F64)[..., None] * inv
            ang = f[0].clone()
            for axis in (1, 2):
                ang[..., axis:60:3] = f[axis][..., axis:60:3]
            ang = ang.reshape(B * T, -1)
        else:
            ang = (torch.arange(T, dtype=F64, device=dev)[:, None] * inv).repeat(B, 1)
        x, aux = _qwen_forward(w, m, x, ang, [T] * B, n, deep)
        x = _rms(x, w["final_norm.weight"])
    mask = batch["loss_mask_BT"][:, 1:].to(F64)
    keep = mask.reshape(-1).nonzero().squeeze(1)
    h = x.view(B, T, -1)[:, :-1].reshape(B * (T - 1), -1)[keep]
    target = ids[:, 1:].reshape(-1)[keep]
    # the head's share of the loss a slice of rows at a time, its gradient at once
    loss, dh, hd = 0.0, [], h.detach()
    for c, t in zip(hd.split(1024), target.split(1024)):
        c = c.requires_grad_()
        part = F.cross_entropy(c @ w["lm_head.weight"].t(), t, reduction="sum") / mask.sum()
        part.backward()
        loss = loss + part.detach()
        dh.append(c.grad)
    torch.autograd.backward([h, aux] if aux.requires_grad else [h], [torch.cat(dh)] + ([torch.ones_like(aux)] if aux.requires_grad else []))
    norm = math.sqrt(sum(float(v.grad.square().sum()) for v in w.values()))
    clip = min(1.0, 1.0 / (norm + 1e-6))
    return {"loss": loss + aux.detach(), "grad_norm": norm, "moments": {k: v.grad.mul_(0.1 * clip) for k, v in w.items()}}


def _letitar_forward(w, x, lengths):
    dev, N, latent = x.device, x.shape[0], {}
    pos = torch.cat([torch.arange(n, dtype=F64, device=dev) for n in lengths])
    # rotation scaled for 8 times 4096 tokens
    freq = 10000.0 ** (-torch.arange(0, 64, 2, dtype=F64, device=dev) / 64)
    pair = lambda turns: 64 * math.log(4096 / (turns * 2 * math.pi)) / (2 * math.log(10000.0))  # noqa: E731
    lo, hi = max(math.floor(pair(16.0)), 0), min(math.ceil(pair(1.0)), 63)
    ramp = ((torch.arange(32, dtype=F64, device=dev) - lo) / max(hi - lo, 0.001)).clamp(0, 1)
    ang, amp = pos[:, None] * (freq / 8 * ramp + freq * (1 - ramp)), 0.1 * math.log(8) + 1
    seq = torch.repeat_interleave(torch.arange(len(lengths), device=dev), torch.tensor(lengths, device=dev))
    for i in range(8):
        p = f"layers.{i}."
        W = lambda key: w[p + key].to(F64)  # noqa: E731
        h = F.layer_norm(x, x.shape[-1:], W("norm1.weight"), W("norm1.bias"), 1e-6)
        proj = h @ W("mixer.in_proj.weight").t()
        if i in (0, 4, 7):
            q = proj[:, :6144].view(N, 32, 192)
            q = torch.cat([q[..., :128], _turn_pairs(q[..., 128:], ang, amp)], -1)
            if i < 7:
                latent[i] = _rms(proj[:, 6144:6656], W("mixer.latent_norm")), _turn_pairs(proj[:, 6656:].view(N, 1, 64), ang, amp)
            c, rot = latent[4 if i == 7 else i]
            k, v = (c @ W("mixer.kv_proj.weight").t()).view(N, 64, 128).split([32, 32], 1)
            y = _attend(q, torch.cat([k, rot.expand(-1, 32, -1)], -1), v, lengths, 192 ** -0.5).reshape(N, -1)
        else:
            q, k, v, gate = (t.view(N, 32, 128) for t in proj[:, : 4 * 4096].split(4096, -1))
            z = proj[:, 4 * 4096:] @ W("mixer.decay_proj.weight").t() + W("mixer.decay_bias")
            alpha = (torch.sigmoid(z) ** (1 / 8.0)).view(N, 32, 128)
            B, T = len(lengths), max(lengths)
            at = (seq, pos.long())
            grid = lambda t, fill: torch.full((B, T, 32, 128), fill, dtype=F64, device=dev).index_put(at, t)  # noqa: E731
            q, k, v, alpha = grid(q * 128 ** -0.5, 0.0), grid(k, 0.0), grid(v, 0.0), grid(alpha, 1.0)
            S, o = x.new_zeros(B, 32, 128, 128), x.new_empty(B, T, 32, 128)
            for t in range(T):
                S.mul_(alpha[:, t, :, :, None]).addcmul_(k[:, t, :, :, None], v[:, t, :, None])
                o[:, t] = (q[:, t, :, None] @ S).squeeze(2)
            y = (_rms(o[at], W("mixer.norm_weight")) * F.silu(gate)).reshape(N, -1)
        x = x + y @ W("mixer.out_proj.weight").t()
        h = F.layer_norm(x, x.shape[-1:], W("norm2.weight"), W("norm2.bias"), 1e-6)
        up, down = W("mlp.up.weight"), W("mlp.down.weight")
        x = x + torch.cat([F.relu(c @ up.t()).square() @ down.t() for c in h.split(16384)])
    return x


def _difedra_forward(w, x, lengths):
    dev, N, first = x.device, x.shape[0], None
    pos = torch.cat([torch.arange(n, dtype=F64, device=dev) for n in lengths])
    freq = 500000.0 ** (-torch.arange(0, 128, 2, dtype=F64, device=dev) / 128)
    keep = ((8192 * freq / (2 * math.pi) - 1) / 3).clamp(0, 1)
    ang = pos[:, None] * ((1 - keep) * freq / 8 + keep * freq)
    for i in range(8):
        p = f"layers.{i}."
        W = lambda key: w[p + key].to(F64)  # noqa: E731
        q, k, v = (_rms(x, W("norm1.weight")) @ W("mixer.in_proj.weight").t()).split([4096, 512, 512], -1)
        wq, wk = W("mixer.qk_norm").split([4096, 512])
        q, k, v = _turn(_rms(q, wq).view(N, 32, 128), ang, 128), _turn(_rms(k, wk).view(N, 4, 128), ang, 128), v.view(N, 4, 128)
        first = v if first is None else first
        if i:
            v = (1 - W("mixer.value_mix")) * v + W("mixer.value_mix") * first
        o = _attend_window(q, k, v, lengths, 128 ** -0.5, 4096, W("mixer.sink"))
        x = x + o.reshape(N, -1) @ W("mixer.out_proj.weight").t()
        h = _rms(x, W("norm2.weight"))
        if i == 0:
            g, u = (h @ W("mlp.gate_up.weight").t()).chunk(2, -1)
            x = x + (F.gelu(g, approximate="tanh") * u) @ W("mlp.down.weight").t()
        else:
            score, idx = torch.sigmoid(h @ W("mlp.router.weight").t()).topk(8, -1)
            x = x + _experts(h, score, idx, w[p + "mlp.experts_gate_up"], w[p + "mlp.experts_down"], True)
    return x


def _attend_window(q, k, v, lengths, scale, window, sink):
    """A query sees the last ``window`` tokens: plain causal rows up to that many, else blocks of queries with their keys."""
    if max(lengths) <= window:
        return _attend(q, k, v, lengths, scale, sink=sink)
    out, at, rep = [], 0, q.shape[1] // k.shape[1]
    for n in lengths:
        for a in range(0, n, 1024):
            b, lo = min(a + 1024, n), max(0, a - window + 1)
            s = q[at + a: at + b].transpose(0, 1) @ k[at + lo: at + b].repeat_interleave(rep, 1).permute(1, 2, 0) * scale
            i, j = torch.arange(a, b, device=q.device)[:, None], torch.arange(lo, b, device=q.device)
            s = s.masked_fill((j > i) | (j <= i - window), -math.inf)
            pr = torch.softmax(torch.cat([s, sink[:, None, None].expand(-1, b - a, 1)], -1), -1)[..., :-1]
            out.append((pr @ v[at + lo: at + b].repeat_interleave(rep, 1).transpose(0, 1)).transpose(0, 1))
        at += n
    return torch.cat(out)


@torch.no_grad()
def _exact_serve(case, seed):
    dev, name, lengths = _device(), case["model"], _lengths(case)
    w = _weights(case, seed)
    ids, more = _rows(case, seed)
    rows = [ids[b, :n] for b, n in enumerate(lengths)]
    if case["do"] == "step":
        rows = [torch.cat([r, more[0, b]]) for b, r in enumerate(rows)]
        lengths = [n + 1 for n in lengths]
    x = w["embedder.weight"][torch.cat(rows).long().to(dev)].to(F64)
    last = torch.tensor(lengths, device=dev).cumsum(0) - 1
    head = (w["embedder.weight"] if name == "difedra" else w["lm_head.weight"]).to(F64)
    if name == "letitar":
        x = _letitar_forward(w, x, lengths)[last]
        x = F.layer_norm(x, x.shape[-1:], w["final_norm.weight"].to(F64), w["final_norm.bias"].to(F64), 1e-6)
        return 25.0 * torch.tanh(x @ head.t() / 25.0)
    if name == "difedra":
        x = _difedra_forward(w, x, lengths)[last]
    else:
        m = QWEN[name]
        pos = torch.cat([torch.arange(n, dtype=F64, device=dev) for n in lengths])
        ang = pos[:, None] * m["theta"] ** (-torch.arange(0, 128, 2, dtype=F64, device=dev) / 128)
        x = _qwen_forward(w, m, x, ang, lengths, _layers(case))[0][last]
    return _rms(x, w["final_norm.weight"].to(F64)) @ head.t()


def exact(case, seed):
    if case["do"] == "train":
        return _exact_train(case, seed)
    return {"logits": _exact_serve(case, seed), "cache": None}        # where a page lies is the allocator's business
