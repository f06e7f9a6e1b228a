"""Prefill passes that build their launch arguments once: the same results as layer by layer, and layer by layer wherever the layers or
the port are not the plain ones."""
import pytest
import torch


def _port(device="cpu", **shape):
    from crosspool_b200.engine.ffn_local import LocalFfnPort
    from crosspool_b200.models import config as mc
    from crosspool_b200.models.weights import random_ffn_weights

    cfg = mc.preset("Qwen/Qwen3-0.6B").with_layers(2)
    return LocalFfnPort, cfg, random_ffn_weights(cfg, 1, device, torch.bfloat16)


def _overridden(kind, port_type, cfg, weights, calls, monkeypatch):
    name = kind.split()[-1]

    def counted(self, *a, **k):
        calls.append(name)
        return getattr(port_type, "_kept_" + name)(self, *a, **k)

    monkeypatch.setattr(port_type, "_kept_" + name, getattr(port_type, name), raising=False)
    if kind.startswith("class"):
        monkeypatch.setattr(port_type, name, counted)
        return port_type(cfg, weights)
    if kind.startswith("subclass"):
        return type("Counted", (port_type,), {name: counted})(cfg, weights)
    port = port_type(cfg, weights)
    monkeypatch.setattr(port, name, lambda *a, **k: counted(port, *a, **k))
    return port


OVERRIDES = [f"{how} {name}" for how in ("class", "subclass", "instance") for name in ("run", "publish_targets", "wait_args")]


@pytest.mark.parametrize("kind", OVERRIDES)
def test_ports_that_answer_in_their_own_way_are_asked(kind, monkeypatch):
    port_type, cfg, weights = _port()
    port = _overridden(kind, port_type, cfg, weights, [], monkeypatch)
    port.act, port.y = torch.zeros(4, cfg.intermediate_size, dtype=torch.bfloat16), torch.zeros(4, cfg.hidden_size, dtype=torch.bfloat16)
    assert port.plain_layers(torch.zeros(4, cfg.hidden_size, dtype=torch.bfloat16), 4) is None


# ---------------------------------------------------------------- on the GPU


def _engine(preset="Qwen/Qwen3-0.6B", layers=3, change=None, port=None):
    from crosspool_b200.engine.atn_engine import AttentionEngine, EngineConfig
    from crosspool_b200.engine.ffn_local import LocalFfnPort
    from crosspool_b200.models import config as mc
    from crosspool_b200.models.weights import random_attention_weights, random_ffn_weights

    cfg = mc.preset(preset).with_layers(layers)
    aw, fw = random_attention_weights(cfg, 1, "cuda", torch.bfloat16), random_ffn_weights(cfg, 1, "cuda", torch.bfloat16)
    if change is not None:
        change(cfg, aw, fw)
    torch.cuda.synchronize()
    return AttentionEngine(cfg, aw, (port or LocalFfnPort)(cfg, fw), EngineConfig(max_batch=4, prefill_chunk=512, max_seq_len=512, use_cuda_graph=False))


def _first_logits(e):
    g = torch.Generator().manual_seed(0)
    for n in (3, 150, 77):
        e.add_request(torch.randint(0, e.cfg.vocab_size, (n,), generator=g).tolist(), 1)
    out = e.step()
    assert len(out) == 3 and not e.has_work
    return e.logits[:3].clone()


def _both(e, monkeypatch):
    """Logits as the engine gives them, layer by layer, and whether the first were those of the plain form."""
    taken, plain = [], e._plain_layers

    def spy(*a):
        taken.append(plain(*a))
        return taken[-1]

    monkeypatch.setattr(e, "_plain_layers", spy)
    got = _first_logits(e)
    monkeypatch.setattr(e, "_plain_layers", lambda *a: False)
    return got, _first_logits(e), taken


@pytest.mark.gpu
@pytest.mark.parametrize("preset", ["Qwen/Qwen3-0.6B", "Qwen/Qwen2.5-0.5B"])      # head norms; projection biases
def test_same_logits_as_layer_by_layer(preset, monkeypatch):
    got, want, taken = _both(_engine(preset), monkeypatch)
    assert taken == [True] and torch.equal(got, want)


def _wider(cfg, aw, fw):
    fw[1].gate_up, fw[1].down = torch.cat([fw[1].gate_up, fw[1].gate_up]), torch.cat([fw[1].down, fw[1].down], 1)


def _biased(cfg, aw, fw):
    fw[2].down_bias = torch.randn(cfg.hidden_size, device="cuda")


def _attention_biased(cfg, aw, fw):
    aw.layers[1].qkv_bias = torch.randn(aw.layers[1].qkv.shape[0], device="cuda")


def _tiled(cfg, aw, fw):
    from crosspool_b200.ops import gemm

    fw[1].gate_up = gemm.tile_weight(fw[1].gate_up)


def _transformed(cfg, aw, fw):
    fw[1].extra["gate_transform"] = (1.0, 1.0, 1.7)


def _pitched(cfg, aw, fw):
    w = aw.layers[1].qkv
    aw.layers[1].qkv = torch.cat([w, torch.zeros_like(w[:, :8])], 1)[:, :w.shape[1]]


@pytest.mark.gpu
@pytest.mark.parametrize("change", [_wider, _biased, _attention_biased, _tiled, _transformed, _pitched])
def test_layers_that_differ_go_one_by_one(change, monkeypatch):
    got, want, taken = _both(_engine(change=change), monkeypatch)
    same = _first_logits(_engine())
    assert taken == [False] and torch.equal(got, want) and (change in (_tiled, _pitched) or not torch.equal(got, same))
    if change is _pitched:
        assert torch.equal(got, same)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", OVERRIDES)
def test_overridden_ports_see_every_layer(kind, monkeypatch):
    calls = []
    e = _engine(port=lambda cfg, fw: _overridden(kind, _port()[0], cfg, fw, calls, monkeypatch))
    _first_logits(e)
    assert len(calls) == 3


@pytest.mark.gpu
@pytest.mark.parametrize("preset,change,built,compared", [("Qwen/Qwen3-0.6B", None, 1, True), ("Qwen/Qwen3-0.6B", _biased, 3, False),
                                                          ("Qwen/Qwen3-30B-A3B", None, 3, False)])
def test_refused_passes_pay_for_no_arguments_of_their_own(preset, change, built, compared, monkeypatch):
    """Launch arguments are built once where the layers are plain and once a layer where the port says at once that they are not,
    without a look at the attention's weights."""
    from crosspool_b200.engine import atn_engine
    from crosspool_b200.ops import attention as A

    e, seen, looks = _engine(preset, change=change), [], []
    args, alike = A.rope_args, atn_engine.alike
    monkeypatch.setattr(A, "rope_args", lambda *a: seen.append(1) or args(*a))
    monkeypatch.setattr(atn_engine, "alike", lambda a, b: looks.append(1) or alike(a, b))
    _first_logits(e)
    assert len(seen) == built and bool(looks) == compared
