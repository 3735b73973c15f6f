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
