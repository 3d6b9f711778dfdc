"""Float32 steps below 256 rows: a request's logits are the same bits whatever else is in the step and however its tokens are cut."""
import pytest
import torch

from infinicore_infer_b200.config import MiniCPMConfig
from infinicore_infer_b200.engine import Engine, StepEntry
from infinicore_infer_b200.weights import write_model_folder

pytestmark = pytest.mark.gpu

# widths from 512 on: the products run on the tensor cores, where the cuts of K set the order of the sums
CONFIG = dict(model_type="minicpm", num_hidden_layers=2, hidden_size=512, num_attention_heads=8, num_key_value_heads=2, intermediate_size=1536, vocab_size=600,
              max_position_embeddings=512, rms_norm_eps=1e-5, rope_theta=10000.0, scale_emb=2.0, scale_depth=1.4, dim_model_base=128, tie_word_embeddings=False)


@pytest.fixture(scope="module")
def engine(tmp_path_factory):
    d = str(tmp_path_factory.mktemp("float32"))
    write_model_folder(MiniCPMConfig.from_dict(CONFIG), d, seed=3, std=0.05, norm_std=0.01)
    return Engine.from_folder(d, dtype=torch.float32, cache_tokens=4096, max_requests=40, max_step_tokens=512)


def _tokens(n, seed):
    return torch.randint(0, CONFIG["vocab_size"], (n,), generator=torch.Generator().manual_seed(seed)).tolist()


def _run(engine, mine, portions, others):
    """Logits of all of ``mine``, run in ``portions``; ``others``: what other requests bring to each of those steps."""
    rows, at = [], 0
    for n in portions:
        entries = [StepEntry(("other", i), _tokens(k, 100 + 7 * i + at), []) for i, k in enumerate(others)]
        entries.insert(len(entries) // 2, StepEntry("mine", mine[at: at + n], list(range(n))))
        rows.append(engine.step(entries))
        at += n
    for r in list(engine.cache.lengths):
        engine.end(r)
    engine.check()
    return torch.cat(rows)


@pytest.mark.parametrize("portions,others", [
    ([60], [190]), ([60], [50, 70]), ([60], [1] * 12), ([60], [1] * 20 + [100]),        # beside prompts, decoding rows, both
    ([5, 50, 5], []), ([1] * 60, []), ([20] + [1] * 40, [1] * 22), ([20] + [1] * 40, [1] * 23), ([59, 1], [40, 1, 30])])
def test_a_request_alone_and_beside_others(engine, portions, others):
    mine = _tokens(60, 1)
    alone = _run(engine, mine, [60], [])
    assert torch.equal(_run(engine, mine, portions, others), alone)


def test_steps_of_many_rows_stay_within_rounding(engine):
    """From 256 rows on the norms and the cuts of K follow the step's rows."""
    mine = _tokens(60, 1)
    alone, many = _run(engine, mine, [60], []), _run(engine, mine, [60], [300])
    # two layers of sums of up to 1,536 terms in another order: some tens of roundings of 2^-24 of the largest logit
    assert (many - alone).abs().max() <= 64 * 2.0 ** -24 * alone.abs().max()
