"""Two runners in one program, each on a stream of its own, with their steps in flight at the same time."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graphs", [True, False])
def test_prompt_steps_of_two_runners_interleave(tmp_path, graphs):
    """The 32-bit products in K slices keep their partial sums in scratch between two launches: each runner's results have
    the bits of the same steps run alone."""
    import mini_llm_b200 as m
    from mini_llm_b200.config.base import EngineConfig
    from mini_llm_b200.engine.runner import ModelRunner, StepEntry
    cfg = dict(architectures=["GPT2LMHeadModel"], model_type="gpt2", n_layer=2, n_embd=512, n_head=8, n_inner=2048,
               vocab_size=1000, n_positions=512, layer_norm_epsilon=1e-5, activation_function="gelu_new", eos_token_id=0)
    m.write_random_model(cfg, 3, str(tmp_path), dtype="float32")
    runners = [ModelRunner(str(tmp_path), EngineConfig(dtype="float32", page_size=16, max_tokens=1024, max_num_seqs=4,
                                                       max_num_batched_tokens=512, use_cuda_graphs=graphs)) for _ in range(2)]
    g = torch.Generator().manual_seed(1)
    steps = [[torch.randint(0, 1000, (n,), generator=g, dtype=torch.int32).numpy() for n in (400, 130, 300, 512)] for _ in range(2)]
    streams = [torch.cuda.Stream() for _ in range(2)]

    def run(which, i, kept):
        with torch.cuda.stream(streams[which]):
            r = object()
            runners[which].add_request(r)
            ids = steps[which][i % 4]
            kept[which].append(runners[which].step([StepEntry(r, ids, [0, len(ids) - 1])]).clone())
            runners[which].finish_request(r)

    torch.cuda.synchronize()
    alone, together = ([], []), ([], [])
    for which in range(2):
        for i in range(24):
            run(which, i, alone)
        torch.cuda.synchronize()
    for i in range(24):
        for which in range(2):
            run(which, i, together)
    torch.cuda.synchronize()
    for which in range(2):
        assert all(torch.equal(a, b) for a, b in zip(alone[which], together[which]))
