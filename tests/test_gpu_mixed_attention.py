"""A pass of single tokens ahead of prompt portions, its attention cut in two, against the same pass uncut and against the 32-bit path."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def config(head_dim, kv_heads, cap):
    return dict(architectures=["Gemma2ForCausalLM"], model_type="gemma2", num_hidden_layers=2, hidden_size=128, num_attention_heads=2 * kv_heads,
                num_key_value_heads=kv_heads, head_dim=head_dim, intermediate_size=256, vocab_size=300, sliding_window=48, query_pre_attn_scalar=head_dim,
                attn_logit_softcapping=cap, final_logit_softcapping=30.0, rms_norm_eps=1e-6, hidden_activation="gelu_pytorch_tanh",
                tie_word_embeddings=True, max_position_embeddings=4096)


@pytest.mark.parametrize("head_dim,kv_heads,cap,singles", [(128, 16, 50.0, 10), (256, 8, 50.0, 19), (128, 16, None, 12)])
def test_cut_in_two(head_dim, kv_heads, cap, singles):
    from kapel_b200.engine import Engine, batch

    rng = np.random.default_rng(3)
    draw = lambda n: rng.integers(0, 300, n).tolist()
    histories = [draw(int(n)) for n in rng.integers(20, 400, singles)]
    steps = [[(f"s{i}", h, []) for i, h in enumerate(histories)],
             [(f"s{i}", draw(1), [0]) for i in range(singles)] + [("p", draw(200), list(range(200)))],
             [(f"s{i}", draw(1), [0]) for i in range(singles)] + [("p", draw(70), list(range(70))), ("r", draw(130), list(range(130)))]]
    whole, taken = batch.StepBatch.mixed_tiles, []

    def run(dtype, cut):
        def mixed(self, *sizes):
            got = whole(self, *sizes) if cut else None
            taken.append(got is not None)
            return got
        batch.StepBatch.mixed_tiles = mixed
        try:
            eng = Engine.random(config(head_dim, kv_heads, cap), seed=1, dtype=dtype, max_tokens=singles * 448 + 512, max_sequences=singles + 2)
            return [eng.step(s).double().cpu() for s in steps][1:]
        finally:
            batch.StepBatch.mixed_tiles = whole

    exact, one = run("float32", False), run("bfloat16", False)
    assert not any(taken)
    two = run("bfloat16", True)
    assert sum(taken) == 4                                   # both layers of both mixed passes
    for e, a, b in zip(exact, one, two):
        off = lambda x: float((x - e).norm() / e.norm())
        assert off(b) <= 1.2 * off(a) + 1e-4, (off(b), off(a))
