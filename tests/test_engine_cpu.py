"""The serving loop's rules on CPU objects: when a recorded decode step serves the next prompt. Nothing is launched; the recording is
a stand-in that counts."""
import pytest
import torch

from ringattention_b200.config import LlamaConfig
from ringattention_b200.models.engine import InferenceEngine
from ringattention_b200.models.llama_infer import LlamaInference


class _Graph:
    def replay(self):
        pass


def _engine(cls=LlamaInference, **kw):
    """An engine whose steps are recorded as stand-ins, with one of them recorded."""
    eng = cls(LlamaConfig.named("llama-tiny"), max_context=256, batch=1, device="cpu", **kw)
    eng.recordings = 0

    def record(body):
        eng.recordings += 1
        return _Graph()

    eng._record = record
    _prompt(eng)
    assert eng.recordings == 1
    return eng


def _prompt(eng, steps=3):
    eng.reset()
    eng.length = 128
    for _ in range(steps):
        eng.decode_step_graph()


def test_a_recorded_step_serves_the_next_prompt_on_one_device():
    eng = _engine()
    _prompt(eng)
    eng.params.p16_rep.mul_(2)  # in place: the step reads what is there
    _prompt(eng)
    assert eng.recordings == 1


def _other_weights(eng):
    eng.params = LlamaInference(LlamaConfig.named("llama-tiny"), max_context=256, device="cpu").params


def _other_storage(eng):
    eng.params.p16_shard = eng.params.p16_shard.clone()


def _storage_swapped_below(eng):
    eng.params.p16_rep.data = eng.params.p16_rep.clone()


def _other_cache(eng):
    eng.v_cache[1] = eng.v_cache[1].clone()


def _other_cache_layout(eng):
    eng.k_cache[0] = eng.k_cache[0][:, :128]


def _theta(eng):
    eng.cfg.rope_theta = 5e5


def _eps(eng):
    eng.cfg.rms_eps = 1e-5


def _sampler(eng):
    eng.sample = lambda logits: logits.argmin(dim=-1)


def _body(eng):
    eng._decode_body = lambda tokens: None


@pytest.mark.parametrize("change", [_other_weights, _other_storage, _storage_swapped_below, _other_cache, _other_cache_layout, _theta, _eps, _sampler, _body])
def test_a_step_is_recorded_anew_after_a_change_between_prompts(change):
    eng = _engine()
    change(eng)
    eng.reset()
    assert not eng._graph_serves()
    _prompt(eng)
    assert eng.recordings == 2


def test_a_sampler_or_a_step_of_a_subclass_is_recorded_for_every_prompt():
    class Sampler(LlamaInference):
        def sample(self, logits):
            return logits.argmin(dim=-1)

    class Step(LlamaInference):
        def _decode_body(self, tokens):
            return super()._decode_body(tokens)

    for cls in (Sampler, Step):
        eng = _engine(cls)
        _prompt(eng)
        _prompt(eng)
        assert eng.recordings == 3


def test_steps_of_a_ring_and_of_streams_are_recorded_for_every_prompt():
    """They hold addresses of buffers that other calls on the ring free when they need larger ones, and of the tails."""
    ring = _engine()
    ring.world = 2
    for eng in (ring, _engine(streams=2)):
        n = eng.recordings
        _prompt(eng, steps=5)
        _prompt(eng, steps=5)
        assert eng.recordings == n + 2


def test_replaced_weights_are_not_kept_alive():
    import weakref

    eng = _engine()
    old = weakref.ref(eng.params.p16_shard)
    _other_weights(eng)
    assert old() is None


def test_default_is_to_record_after_every_reset():
    class Engine(InferenceEngine):
        def _clear_cache(self):
            pass

    eng, n = Engine(1, "cpu", 1), []
    eng._record = lambda body: n.append(1) or _Graph()
    for _ in range(3):
        _prompt(eng)
    assert len(n) == 3


def test_a_replayed_step_stands_behind_the_tokens_of_a_step_before_it():
    """The position on the device is written again whenever something else than a replay has moved it, also when the tokens between
    lead back to the place of the last replay."""
    from ringattention_b200.models import registry
    from ringattention_b200.models.hybrid_infer import HybridInference

    eng = HybridInference(registry.load_config("kalonex-tiny"), max_context=64, device="cpu")
    eng._forward = lambda *a, **k: None
    at = []

    class Graph:  # a recorded step advances the position itself
        def replay(self):
            at.append(int(eng.state[0]))
            eng.state[0] += 1

    eng._record = lambda body: Graph()
    tok = torch.zeros(1, 4, dtype=torch.int64)
    eng.step(tok)
    eng.decode_step_graph()
    eng.decode_step_graph()
    eng.length = 2
    eng.step(tok)
    eng.decode_step_graph()
    assert at == [4, 5, 6] and eng.length == 7


@pytest.mark.parametrize("free,fails,emptied", [(1 << 30, 0, 0), ((1 << 30) - 1, 0, 1), (1 << 34, 1, 1), (0, 1, 2), (1 << 34, 2, 1)])
def test_the_allocators_cache_is_emptied_when_a_recording_is_short_of_memory(free, fails, emptied, monkeypatch):
    """A capture cannot make the allocator give its cached blocks back: with too little free memory that happens ahead of it, and after
    one that ran out of memory; a second failure is the caller's."""
    eng, log = InferenceEngine(1, "cpu", 1), []
    monkeypatch.setattr(torch.cuda, "synchronize", lambda *a: None)
    monkeypatch.setattr(torch.cuda, "mem_get_info", lambda device=None: (free, 1 << 37))
    monkeypatch.setattr(torch.cuda, "empty_cache", lambda: log.append("empty"))

    def capture(body):
        log.append("capture")
        if log.count("capture") <= fails:
            raise torch.OutOfMemoryError("no memory")
        return _Graph()

    eng._capture, eng._old_graph = capture, _Graph()
    if fails == 2:
        with pytest.raises(torch.OutOfMemoryError):
            eng._record(None)
    else:
        assert isinstance(eng._record(None), _Graph) and eng._old_graph is None
    assert log.count("empty") == emptied and log.count("capture") == 1 + min(fails, 1)
    assert log[0] == ("empty" if free < 1 << 30 else "capture")
