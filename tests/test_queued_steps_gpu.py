"""Mixed steps queued behind one another: a step's decoding requests and its prompt portion are attended by two kernels in a row, each
of which must find what the kernels before them wrote."""
import pytest
import torch

pytestmark = pytest.mark.gpu

RAW = {"architectures": ["Qwen2ForCausalLM"], "model_type": "qwen2", "hidden_size": 1792, "num_attention_heads": 14,
       "num_key_value_heads": 2, "head_dim": 128, "intermediate_size": 4864, "num_hidden_layers": 4, "vocab_size": 4096,
       "rope_theta": 1000000.0, "rms_norm_eps": 1e-6, "tie_word_embeddings": False}
CONTEXTS, PORTION, AT = (100, 131, 257, 700, 901, 64, 15, 333), 617, 130


def test_queued_mixed_steps_repeat_themselves():
    from blackwellllm_b200 import Engine, StepEntry
    gen = torch.Generator().manual_seed(3)
    ids = lambda n: torch.randint(0, 4096, (n,), generator=gen).tolist()
    engines = [Engine.from_config(RAW, seed=s, num_pages=260, max_requests=10, max_batch_tokens=1024, max_context=1024) for s in (0, 1)]
    lengths = dict(enumerate(CONTEXTS), p=AT)
    prompts, step_ids = {r: ids(n) for r, n in lengths.items()}, ids(len(CONTEXTS) + PORTION)
    for e in engines:
        for r, tokens in prompts.items():
            e.step([StepEntry(r, tokens, [])])
    entries = [StepEntry(r, [step_ids[r]], [0]) for r in range(len(CONTEXTS))]
    entries.append(StepEntry("p", step_ids[len(CONTEXTS):], [0, 300, PORTION - 1]))

    def step(e):
        logits = e.step(entries)
        for r, n in lengths.items():
            e.cache.truncate(r, n)
        return logits

    alone = []
    for e in engines:
        for _ in range(2):
            torch.cuda.synchronize()
            logits = step(e)
            torch.cuda.synchronize()
        alone.append(logits)
    assert not torch.equal(*alone)
    for _ in range(8):
        queued = [step(engines[i % 2]) for i in range(50)]
        assert all(torch.equal(out, alone[i % 2]) for i, out in enumerate(queued))


def test_two_mixers_as_branches_of_a_graph():
    """A recorded step runs the two mixers beside each other; its bits are those of uncaptured steps, also of many steps queued."""
    import tiny_zanivik
    from blackwellllm_b200 import Engine, StepEntry
    raw, page = tiny_zanivik.CONFIGS["broad"]
    weights = {n: t.cuda() for n, t in tiny_zanivik.make_tensors(raw, 5).items()}
    got = []
    for graphs in (False, True):
        e = Engine.from_tensors(raw, weights, dtype="bfloat16", page_size=page, num_pages=40, max_requests=6, max_batch_tokens=512,
                                max_context=512, cuda_graphs=graphs)
        for r in range(6):
            e.step([StepEntry(r, tiny_zanivik.prompt(20 + 37 * r, raw["vocab"], r), [])])
        logits = []
        for s in range(60):
            # (a replay's logits are overwritten by the next one)
            logits.append(e.step([StepEntry(r, [(31 * s + 7 * r) % raw["vocab"]], [0]) for r in range(6)]).clone())
        got.append(torch.stack(logits))
        assert bool(e.graph_kernel_count(6)) == graphs
    assert torch.equal(*got)
