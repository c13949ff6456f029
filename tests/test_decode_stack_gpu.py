"""The one-launch decode step (csrc/decode_stack.cu) beside the step layer by layer: the same engine with IMP_B200_DECODE_STACK 1 and 0.
Both round to bfloat16 at the same places and differ in the order of 32-bit sums alone, so against the plain implementation in
float32 neither may be much further away than the other: at most 1.25 times as far, the spread of a maximum over a few rows of rounding errors."""
import numpy as np
import pytest

from plain.qwen3_plain import PlainModel

pytestmark = pytest.mark.gpu

BASE = {"architectures": ["Qwen3ForCausalLM"], "vocab_size": 509, "num_hidden_layers": 2, "head_dim": 128, "rms_norm_eps": 1e-6, "rope_theta": 1e6,
        "tie_word_embeddings": True, "torch_dtype": "bfloat16", "max_position_embeddings": 1024}
# width, query heads, kv heads, inner size: fewer columns than CTAs; a last part of the contraction of 64; groups of 8 heads, one, five;
# shares of more than one tile and of two parts (1,088 = 1,024 + 64); inner sizes of several parts (3,136, 2,048)
SHAPES = [(64, 2, 2, 64), (192, 8, 1, 320), (1088, 5, 1, 3136), (1024, 4, 2, 2048), (2560, 16, 8, 704)]
# lengths before the single tokens: around the 16 and 32 keys of a run and a block, and enough for several parts of the keys
LENGTHS = [[1], [15], [31, 32, 33], [16, 130, 700], [1, 2, 31, 63, 64, 65, 127, 300]]


def replay(folder, lengths, ids, page, stacked, monkeypatch):
    from imp_b200 import Engine, EngineConfig, StepEntry
    monkeypatch.setenv("IMP_B200_DECODE_STACK", "1" if stacked else "0")
    eng = Engine.from_folder(folder, EngineConfig(max_batch_size=8, max_seq_len=1024, kv_cache_max_blocks=8 * 1024 // page, kv_block_size=page,
                                                  max_batch_tokens=1024, compute_dtype="bfloat16"))
    for r, n in enumerate(lengths):
        eng.step_tokens([StepEntry(r, ids[r][:n], [])])
    rows, launches = [], []
    for k in range(4):       # eager, captured, replayed twice
        before = eng.info()["launches"]
        rows.append(eng.step_tokens([StepEntry(r, [ids[r][n + k]], [0]) for r, n in enumerate(lengths)]).copy())
        launches.append(eng.info()["launches"] - before)
    eng.close()
    return np.stack(rows, 1), launches      # [sequence, step, vocab]


@pytest.fixture(scope="module", params=SHAPES, ids=str)
def model(request, tmp_path_factory):
    from imp_b200 import config_from_dict, write_model_folder
    d, hq, hkv, f = request.param
    folder = str(tmp_path_factory.mktemp("stack"))
    write_model_folder(folder, config_from_dict(dict(BASE, hidden_size=d, num_attention_heads=hq, num_key_value_heads=hkv, intermediate_size=f)), seed=5,
                       std=0.64 / d ** 0.5)
    return folder, PlainModel(folder)


@pytest.mark.parametrize("page", [16, 64])
@pytest.mark.parametrize("lengths", LENGTHS, ids=str)
def test_one_launch_gives_the_layers_logits(model, lengths, page, monkeypatch):
    folder, plain = model
    rng = np.random.default_rng(len(lengths))
    ids = [rng.integers(0, BASE["vocab_size"], n + 4).tolist() for n in lengths]
    want = np.stack([plain.logits(v)[-4:].numpy() for v in ids]).astype(np.float64)
    apart, n_apart = replay(folder, lengths, ids, page, False, monkeypatch)
    one, n_one = replay(folder, lengths, ids, page, True, monkeypatch)
    assert max(n_one) <= 6 < min(n_apart)     # embedding, layers, norm, head (and its sum): not layer by layer
    err = [np.linalg.norm((x - want).reshape(len(lengths), -1), axis=1) / np.linalg.norm(want.reshape(len(lengths), -1), axis=1) for x in (one, apart)]
    assert np.isfinite(one).all() and err[0].max() <= 1.25 * err[1].max() + 1e-4, err


def test_more_tokens_than_the_launch_takes_go_layer_by_layer(model, monkeypatch):
    from imp_b200 import Engine, EngineConfig, StepEntry
    folder, _ = model
    monkeypatch.setenv("IMP_B200_DECODE_STACK", "1")
    eng = Engine.from_folder(folder, EngineConfig(max_batch_size=9, max_seq_len=64, kv_cache_max_blocks=64, kv_block_size=16, max_batch_tokens=64,
                                                  compute_dtype="bfloat16"))
    counts = []
    for n in (8, 9, 8):
        before = eng.info()["launches"]
        eng.step_tokens([StepEntry(r, [r + 1], [0]) for r in range(n)])
        counts.append(eng.info()["launches"] - before)
    eng.close()
    assert counts[0] == counts[2] < counts[1]
