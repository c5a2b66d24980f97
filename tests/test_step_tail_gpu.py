"""Steps that follow one another on the device: the kernel behind the sampling, and requests whose sequences cross page borders,
end at different times and change batches, against steps laid out one by one."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("n", [1, 5, 256, 300])
def test_step_tail(n):
    from gguf_rs_cli_b200 import kernels as k
    i32 = dict(dtype=torch.int32, device=DEV)
    out, tokens, pos, starts = [torch.randint(0, 1000, (n,), **i32) for _ in range(4)]
    seq_of = torch.arange(n, **i32)
    seq_of[n // 2:n // 2 + 1 + n // 7] = -1
    live = (seq_of >= 0).int()
    want = torch.where(live > 0, out, tokens), pos + live, starts + live, pos + 2 * live
    hosts, turn = [torch.full((n + 3,), -7, dtype=torch.int32).pin_memory() for _ in range(2)], torch.zeros(1, **i32)
    k.step_tail(out, seq_of, tokens, pos, starts, turn, hosts)
    torch.cuda.synchronize()
    assert torch.equal(tokens, want[0]) and torch.equal(pos, want[1]) and torch.equal(starts, want[2]) and turn.item() == 1
    assert hosts[0][:n].tolist() == out.tolist() and (hosts[0][n:] == -7).all() and (hosts[1] == -7).all()
    out += 1
    k.step_tail(out, seq_of, tokens, pos, starts, turn, hosts)
    torch.cuda.synchronize()
    assert hosts[1][:n].tolist() == out.tolist() and hosts[0][:n].tolist() == (out - 1).tolist() and turn.item() == 0 and torch.equal(pos, want[3])


@pytest.mark.parametrize("lens, n", [([60, 61, 3], 140), ([64], 70), ([1, 128, 63, 127, 2], 80)])
def test_requests_over_page_borders_are_those_of_steps_one_by_one(lens, n):
    """Captured steps that feed themselves give the ids of eager steps, whose index arrays come from the host every time: over page
    borders, with a stop token that ends some sequences early (the batch shrinks), twice on the same engine."""
    from gguf_rs_cli_b200.engine.backend import EngineBackend
    from gguf_rs_cli_b200.engine.generate import generate_ids
    from gguf_rs_cli_b200.sampling.params import SamplingParams
    from tests.test_model_gpu import new_engine, tokens_of
    prompts = [tokens_of("A", m, 100 + i) for i, m in enumerate(lens)]
    got = []
    for graphs in (False, True):
        backend = EngineBackend(new_engine("A", "bfloat16", n_tokens=64 * 32, n_slots=8), use_graphs=graphs)
        runs = []
        for params, stops in ((SamplingParams(temperature=0.0), ()), (SamplingParams(temperature=0.9, top_k=20, seed=3), ()),
                              (SamplingParams(temperature=0.9, top_k=20, seed=3), None), (SamplingParams(temperature=0.0), ())):
            if stops is None:                       # ids that the run before has drawn in the middle of its first and last sequence
                stops = (runs[-1][0][30], runs[-1][-1][45])
            runs.append(generate_ids(backend, prompts, n, params, stop_token_ids=stops))
        got.append(runs)
        assert not graphs or backend.steps_ahead > n
    assert got[0] == got[1] and got[1][0] == got[1][3]
