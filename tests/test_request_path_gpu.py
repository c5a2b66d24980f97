"""The host path of a request on the device: the engine that is kept between calls, and the index arrays of a step."""
import pytest
import torch

from tests.gpu_util import llm, new_engine, tokens_of

pytestmark = pytest.mark.gpu


def _fresh(name, dtype, prompts, **kw):
    from gguf_rs_cli_b200.api import generate
    model = llm(name, dtype)
    model._engine = model._backend = None
    return generate(model, prompts, stop_token_ids=[], **kw)


# 5 + 59 = 64 positions fill a page to its end: no engine may end such a sequence early
@pytest.mark.parametrize("shape", [((5, 9, 13), 8), ((70, 3), 30), ((5,), 59), ((5, 64), 64)])
def test_a_kept_engine_answers_as_a_new_one(shape):
    from gguf_rs_cli_b200.api import generate
    lens, n = shape
    prompts = [tokens_of("C", k, 300 + k) for k in lens]
    want = _fresh("C", "float32", prompts, max_tokens=n)
    assert [len(w) for w in want] == [n] * len(lens)
    model = llm("C", "float32")
    made = model._engine
    assert generate(model, prompts, max_tokens=n, stop_token_ids=[]) == want and model._engine is made
    # a smaller call is served by the same engine
    small = [p[:4] for p in prompts]
    got = generate(model, small, max_tokens=n, stop_token_ids=[])
    assert model._engine is made and [len(g) for g in got] == [n] * len(lens)
    assert got == _fresh("C", "float32", small, max_tokens=n)
    # and both by one that holds the model's longest sequence
    generate(model, [tokens_of("C", 900, 9)] * 3, max_tokens=124, stop_token_ids=[])
    made = model._engine
    assert made.cache.max_len == model.spec.max_position
    assert generate(model, prompts, max_tokens=n, stop_token_ids=[]) == want
    assert generate(model, small, max_tokens=n, stop_token_ids=[]) == got and model._engine is made


def test_graphs_that_are_kept_are_bounded():
    from gguf_rs_cli_b200.engine.backend import EngineBackend
    from gguf_rs_cli_b200.engine.generate import generate_ids
    from gguf_rs_cli_b200.sampling import SamplingParams
    backend = EngineBackend(new_engine("A", "float32", n_tokens=256, n_slots=2))
    backend.MAX_GRAPHS = 2
    prompt = [tokens_of("A", 6, 1)]
    want = generate_ids(backend, prompt, 6, SamplingParams(temperature=0.5, seed=1), [])
    for t in (0.6, 0.7, 0.8):
        generate_ids(backend, prompt, 6, SamplingParams(temperature=t, seed=1), [])
        assert len(backend._graphs) <= 2
    assert generate_ids(backend, prompt, 6, SamplingParams(temperature=0.5, seed=1), []) == want


@pytest.mark.parametrize("n", [7, 200])                  # laid out as lists, and as arrays
@pytest.mark.parametrize("kind", ["list", "numpy", "tensor", "int32", "bool"])
def test_token_ids_of_every_kind(kind, n):
    import numpy as np
    from gguf_rs_cli_b200.engine.step import Entry, StepError
    ids = tokens_of("C", n, 2)
    make = {"list": list, "numpy": np.asarray, "tensor": torch.tensor, "int32": lambda x: np.asarray(x, np.int32),
            "bool": lambda x: [bool(t % 2) for t in x]}[kind]
    plain = [int(t) for t in make(ids)]
    eng = new_engine("C", "float32", n_tokens=1024, n_slots=3)
    s = [eng.open() for _ in range(3)]
    a = eng.step([Entry(s[0], plain, (n - 1,))]).clone()
    b = eng.step([Entry(s[1], make(ids), (n - 1,))])
    assert torch.equal(a, b)
    if kind != "bool":
        with pytest.raises(StepError, match="outside the vocabulary"):
            eng.step([Entry(s[2], make(ids[:-1] + [1000]), ())])
        with pytest.raises(StepError, match="outside the vocabulary"):
            eng.step([Entry(s[2], make([-1] + ids), ())])


def test_an_interrupted_request_leaves_nothing_in_flight():
    """... and the next one, on another stream, has its buffers to itself."""
    from gguf_rs_cli_b200.api import generate
    prompts = [tokens_of("C", k, 400 + k) for k in (90, 40)]
    want = _fresh("C", "bfloat16", prompts, max_tokens=20)
    model = llm("C", "bfloat16")
    made = model._engine

    def boom(request, token):
        if len(seen) == 9:
            raise RuntimeError("callback")
        seen.append(token)
    for _ in range(3):
        seen = []
        with pytest.raises(RuntimeError, match="callback"):
            generate(model, prompts, max_tokens=20, stop_token_ids=[], on_token=boom)
        assert torch.cuda.current_stream().query()
        with torch.cuda.stream(torch.cuda.Stream()):
            assert generate(model, prompts, max_tokens=20, stop_token_ids=[]) == want and model._engine is made
            torch.cuda.synchronize()


@pytest.mark.parametrize("at", [1, 2, 3, 4, 5, 6, 9, 26, 27])
def test_a_request_interrupted_behind_a_launch_leaves_the_next_ones_ids(at):
    """The interruption comes when the device has the step and the host has not counted it: behind the prompts' step, the eager step,
    the captured one, those that follow on the device and those of a page border (lengths 90 and 40: the step behind 64 and 128 tokens)."""
    from gguf_rs_cli_b200.api import generate
    from gguf_rs_cli_b200.engine.backend import EngineBackend
    prompts = [tokens_of("C", k, 400 + k) for k in (90, 40)]
    want = _fresh("C", "bfloat16", prompts, max_tokens=40)
    model = llm("C", "bfloat16")
    for warm in (False, True):
        if not warm:                               # nothing is captured; then everything is
            model._engine = model._backend = None
        calls, real = [], EngineBackend._pending

        def boom(self, *args, **kw):
            calls.append(1)
            if len(calls) == at:
                raise KeyboardInterrupt
            return real(self, *args, **kw)
        with pytest.MonkeyPatch.context() as m:
            m.setattr(EngineBackend, "_pending", boom)
            with pytest.raises(KeyboardInterrupt):
                generate(model, prompts, max_tokens=40, stop_token_ids=[])
        for _ in range(2):
            assert generate(model, prompts, max_tokens=40, stop_token_ids=[]) == want


@pytest.mark.parametrize("lens", [[1] * 130, [1, 200, 1, 33, 5, 129, 32], [40, 3], [2] * 70 + [129] + [1] * 3, [33] * 5])
def test_index_arrays_of_long_and_short_sequences_side_by_side(lens):
    """Laid out as arrays, as lists and as both in turn: in 32-bit mode every sequence's logits are those of a step of its own."""
    from gguf_rs_cli_b200.engine.step import Entry
    eng = new_engine("C", "float32", n_tokens=sum((n + 63) // 64 * 64 for n in lens), n_slots=len(lens))
    prompts = [tokens_of("C", n, 500 + k) for k, n in enumerate(lens)]
    slots = [eng.open() for _ in lens]
    together = eng.step([Entry(s, p, (len(p) - 1,)) for s, p in zip(slots, prompts)]).clone()
    for s in slots:
        eng.close(s)
    for row, p in list(zip(together, prompts))[::7] + [(together[-1], prompts[-1])]:
        s = eng.open()
        assert torch.equal(row, eng.step([Entry(s, p, (len(p) - 1,))])[0])
        eng.close(s)


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_a_captured_step_allocates_nothing(dtype):
    """Of matrices that are large enough for the tensor cores in either type: all buffers are there before the capture."""
    from gguf_rs_cli_b200.api import _build
    from gguf_rs_cli_b200.engine.backend import EngineBackend
    from gguf_rs_cli_b200.engine.generate import generate_ids
    from gguf_rs_cli_b200.engine.step import Engine
    from gguf_rs_cli_b200.weights import TensorSource
    from tests import plain_llama as P
    from tests.tiny import config
    raw = dict(config("A"), hidden_size=1024, num_attention_heads=16, num_key_value_heads=4, head_dim=64, intermediate_size=2048, num_hidden_layers=1)
    w = {k: v.to(getattr(torch, dtype)) for k, v in P.random_weights(raw, 0).items()}
    model = _build(raw, TensorSource(tensors=w, where="one layer"), dtype, "cuda:0")
    backend, seen = EngineBackend(Engine(model.model, n_tokens=256, n_slots=2)), []
    real = backend._capture

    def counted(body):
        allocated = lambda: torch.cuda.memory_stats()["allocation.all.allocated"]

        def inside():
            before = allocated()
            body()
            seen.append(allocated() - before)
        return real(inside)
    backend._capture = counted
    for n in (1, 2):
        prompts = [tokens_of("A", 5, i) for i in range(n)]
        assert len(generate_ids(backend, prompts, 6)) == n
    assert seen == [0] * len(seen) and len(seen) >= 2
