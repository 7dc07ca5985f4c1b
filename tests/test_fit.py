"""The forecast of the memory a model takes (weights, cache, scratch) and the refusal before anything is
allocated."""
import pytest
import torch

from helpers import TINY, cpu_model, model_folder


def test_forecast_counts_what_is_allocated():
    m = cpu_model("B", "float32", max_tokens=640)
    fc = m.forecast(640)
    cfg = TINY["B"]
    # weights: every tensor of the plan; float32 path keeps 4 bytes per element
    plan_bytes = 0
    for spec in m.plan().values():
        n = 1
        for d in spec.shape:
            n *= d
        plan_bytes += n * 4
    assert fc.weights == plan_bytes
    # cache: layers x pages x (k, v) x kv heads x 64 x head_dim x 4 bytes; the model's cache holds exactly that
    pages = 640 // 64
    assert fc.cache == cfg["num_hidden_layers"] * pages * 2 * cfg["num_key_value_heads"] * 64 * cfg["head_dim"] * 4
    from cima_b200.sampling import sampler_state
    with_state = m.forecast(640, extra_state=sampler_state())      # as load_model asks: the sampler's state per slot
    assert with_state.cache == (sum(g.nbytes() for g in m.cache.groups)
                                + sum(t.numel() * t.element_size() for t in m.cache.state.values()))
    assert fc.scratch > 0 and fc.total == fc.weights + fc.cache + fc.scratch
    assert "GiB" in fc.describe()
    half = cpu_model("B", "bfloat16", max_tokens=640).forecast(640)
    assert half.cache * 2 == fc.cache          # bfloat16 keys and values


def test_forecast_counts_the_segments_of_a_long_steps_recurrence():
    """Two states (and a column of one) for every 128 rows of the largest step, of the mixer with the largest state; bfloat16 only,
    as 32-bit sequences are not cut."""
    import gisirax_cases
    from cima_b200.engine import fit
    m = gisirax_cases.cpu_model("C", "bfloat16", max_tokens=640)
    seen = {}
    plain, fit.forecast = fit.forecast, lambda *a, **kw: (seen.update(kw), plain(*a, **kw))[1]
    try:
        with_segments = m.forecast(20000)
    finally:
        fit.forecast = plain
    rights = [l["mixer"]["right"] for l in gisirax_cases.CONFIGS["C"]["layers"] if l["type"] == "parallel"]
    row = max(2.0 * r["heads"] * r["dim"] * (r["vdim"] + 1) * 4 / 128 for r in rights)
    assert seen["segment_row"] == row
    args = (m.plan(), m._cache_requests(), torch.bfloat16, 20000, 256, 640, 512)
    assert plain(*args, segment_row=row).scratch - plain(*args).scratch == int(fit.STEP_ROWS * row)
    assert with_segments.scratch > plain(*args).scratch
    seen.clear()
    fit.forecast = lambda *a, **kw: (seen.update(kw), plain(*a, **kw))[1]
    try:
        gisirax_cases.cpu_model("C", "float32", max_tokens=640).forecast(640)
    finally:
        fit.forecast = plain
    assert seen["segment_row"] == 0.0


@pytest.mark.gpu
def test_recorded_one_token_steps_stay_within_their_part_of_the_forecast():
    """Steps of 33 to 48 sequences recorded, sixteen of them: the memory that stays taken is their logits and one step's activations
    (and what the allocator rounds up to, blocks of 20 MiB), as the forecast has it."""
    import cima_b200
    from cima_b200.config.shapes import SHAPES
    from cima_b200.engine import StepEntry
    from cima_b200.engine.graph import MAX_STEP_GRAPHS
    lm = cima_b200.load(config=dict(SHAPES["qwen2.5-0.5b"], num_hidden_layers=2), draw="device", max_tokens=64 * 64, max_seqs=64, verbose=False)
    slots = lm.model.cache.open(48)
    lm.step([StepEntry(s, [1, 2], [1]) for s in slots])
    for n in range(33, 49):                              # (a size's first step needs what a step needs)
        lm.step([StepEntry(s, [3], [0]) for s in slots[:n]])
    torch.cuda.synchronize(); torch.cuda.empty_cache()
    before = torch.cuda.memory_reserved()
    for n in range(33, 49):
        lm.step([StepEntry(s, [4], [0]) for s in slots[:n]])
        lm.step([StepEntry(s, [5], [0]) for s in slots[:n]])
    torch.cuda.synchronize(); torch.cuda.empty_cache()
    assert len(lm.model._step_graphs) == MAX_STEP_GRAPHS and all(g.graph is not None for g in lm.model._step_graphs.values())
    vocab, row = lm.spec.vocab, 896 * 4 + (2 * 4864 + 2 * 896) * 2
    assert torch.cuda.memory_reserved() - before <= 64 * (MAX_STEP_GRAPHS * vocab * 4 + row)
    from cima_b200.engine import fit
    m, held = lm.model, fit.forecast
    plan = (m.plan(), m._cache_requests(), torch.bfloat16, 4096, 896, vocab, 2 * 4864)
    assert held(*plan, max_seqs=64).scratch - held(*plan, max_seqs=63).scratch == MAX_STEP_GRAPHS * vocab * 4 + row + 2 * vocab * 4


@pytest.mark.gpu
def test_a_cache_that_cannot_fit_is_refused_before_allocating():
    from cima_b200.engine import load_model
    from cima_b200.engine.fit import DoesNotFit
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    with pytest.raises(DoesNotFit, match="does not fit"):
        load_model(model_folder("B"), dtype="bfloat16", max_tokens=10 ** 10, device="cuda:0", verbose=False)
    assert torch.cuda.memory_allocated() == before


def test_how_far_prompt_steps_are_recorded_follows_the_model_size():
    """A recorded prompt step pays while the device finishes its padded rows before the host could have issued the
    launches: the known shapes land where they were measured to (0.5B wins up to 2,048 rows, 1.5B up to 768, 3B up to
    512 or 768, 7B and larger only within the 256 rows that every model gets)."""
    from cima_b200.config.shapes import SHAPES
    from cima_b200.engine.graph import PROMPT_ROWS, recorded_prompt_rows

    def step_bytes(c):
        H, I, L = c["hidden_size"], c["intermediate_size"], c["num_hidden_layers"]
        qkv = (c["num_attention_heads"] + 2 * c["num_key_value_heads"]) * c["head_dim"]
        return 2 * (L * (H * qkv + c["num_attention_heads"] * c["head_dim"] * H + 3 * H * I) + c["vocab_size"] * H)

    got = {name: recorded_prompt_rows(step_bytes(SHAPES[name]), SHAPES[name]["num_hidden_layers"], 2)
           for name in ("qwen2.5-0.5b", "qwen2.5-1.5b", "qwen2.5-3b", "qwen2.5-7b", "qwen2.5-32b")}
    assert got == {"qwen2.5-0.5b": 2048, "qwen2.5-1.5b": 768, "qwen2.5-3b": 512, "qwen2.5-7b": PROMPT_ROWS,
                   "qwen2.5-32b": PROMPT_ROWS}
    assert recorded_prompt_rows(1e6, 2, 4) == 2048 and recorded_prompt_rows(1e12, 2, 2) == PROMPT_ROWS
