"""One launch or three for decode attention over shared prompts: the rule against what was measured on a B200."""
import numpy as np
import pytest

from arctic_platform_b200.ops.forest_attention import one_launch_pays

# query heads, key heads, prompts, samples, shared tokens, own tokens (negative: uniform up to twice that), share of live slots, three, one (us)
MEASURED = [
    (32, 8, 8, 16, 2048, 17, 1.0, 46.8, 26.6), (32, 8, 8, 16, 2048, 512, 1.0, 84.1, 74.0), (32, 8, 8, 16, 2048, 2048, 1.0, 194.0, 209.7),
    (32, 8, 8, 16, 2048, -128, 1.0, 55.1, 45.4), (32, 8, 8, 16, 2048, -512, 1.0, 82.5, 101.3), (32, 8, 8, 16, 2048, -1024, 0.1, 58.9, 84.4),
    (32, 8, 1, 16, 2048, 256, 1.0, 24.7, 20.1), (32, 8, 1, 16, 2048, 2048, 1.0, 45.3, 59.2), (32, 8, 1, 4, 512, 1024, 1.0, 19.1, 21.9),
    (32, 8, 4, 8, 512, 512, 1.0, 28.6, 24.1), (32, 8, 40, 4, 512, 17, 1.0, 64.7, 56.7), (32, 8, 40, 4, 512, 256, 1.0, 84.3, 102.3),
    (32, 8, 64, 2, 1024, 1024, 1.0, 184.1, 165.7), (32, 8, 1, 8, 16384, 2048, 1.0, 98.0, 48.2), (16, 8, 1, 8, 512, 2048, 1.0, 25.3, 35.3),
    (32, 4, 4, 8, 512, 2048, 1.0, 42.5, 50.5), (32, 4, 8, 16, 2048, 128, 1.0, 38.5, 26.2),
    (16, 4, 1, 32, 416, 8, 1.0, 17.1, 24.4), (16, 8, 64, 16, 256, 17, 1.0, 153.4, 250.8), (32, 8, 16, 32, 2048, 17, 1.0, 117.2, 80.4),
    (32, 8, 1, 16, 2048, 17, 1.0, 21.2, 18.8), (64, 8, 4, 16, 3728, 15, 1.0, 42.1, 33.8),
]


@pytest.mark.parametrize("case", MEASURED)
def test_the_faster_form_is_chosen(case):
    """Sizes whose two times differ by more than the sums of the rule are off."""
    Hq, Hkv, prompts, samples, shared, own, live, three, one = case
    B, rng, sms = prompts * samples, np.random.default_rng(0), 148
    tokens = np.full(B, own) if own > 0 else rng.integers(1, -2 * own, B)
    rng.permutation(B * ((int(tokens.max()) + 15) // 16 + 1))            # of the pages, in what was measured
    tokens[rng.permutation(B)[int(B * live):]] = 0
    tile = 128 * Hkv // Hq
    runs = prompts * -(-samples // tile)
    node_rows = 1 << (runs - 1).bit_length()
    room, fit = sms // (node_rows * Hkv), max(4 * B, 256) // B
    got = one_launch_pays(np.full(runs, shared), np.full(runs, min(samples, tile)), tokens, np.zeros(B), node_rows, Hq, Hkv, max(1, min(8, fit, room)),
                          min(64, fit), max(1, min(4, room)), max(1, min(4, 296 // (B * Hkv))), sms)
    assert got == (one < three)


@pytest.mark.parametrize("B,Hkv,nodes", [(1, 1, 1), (8, 8, 16), (300, 2, 3), (1024, 1, 512)])
def test_any_batch_has_an_answer(B, Hkv, nodes):
    """No tokens, one slot, more slots than the kernel looks for better parts at, nodes of no tokens."""
    for own in (np.zeros(B, dtype=np.int64), np.arange(B), np.full(B, 100000)):
        for splits in (1, 8):
            assert one_launch_pays(np.zeros(min(nodes, 3), dtype=np.int32), np.ones(min(nodes, 3), dtype=np.int32), own, own[::-1], nodes, 8 * Hkv, Hkv,
                                   splits, 4, 4, 1, 148) in (True, False)
    with pytest.raises(ValueError, match="out of range"):
        one_launch_pays(np.zeros(2), np.ones(2), np.ones(B), np.ones(B), 1, 8 * Hkv, Hkv, 1, 4, 4, 1, 148)


@pytest.mark.parametrize("prompts,samples,shared,left,one", [(8, 16, 2048, 33, True), (8, 16, 2048, 2047, True), (40, 4, 512, 17, True),
                                                            (40, 4, 512, 1024, False), (8, 16, 2048, 8000, False)])
def test_the_choice_is_for_the_steps_ahead(prompts, samples, shared, left, one):
    """From the first token on: what is saved while responses are short is set against what is lost when they are long.  A slot that has
    no steps left counts as idle."""
    B, sms = prompts * samples, 148
    rows = 1 << (prompts - 1).bit_length()
    room, fit = sms // (rows * 8), max(4 * B, 256) // B
    sizes = (rows, 32, 8, max(1, min(8, fit, room)), min(64, fit), max(1, min(4, room)), max(1, min(4, 296 // (B * 8))), sms)
    runs = np.full(prompts, shared), np.full(prompts, samples)
    assert one_launch_pays(*runs, np.full(B, 1), np.full(B, left), *sizes) == one
    long = np.full(B, 1)
    long[::2] = 5000
    ends = np.where(long > 1, -7, left)
    assert one_launch_pays(*runs, long, ends, *sizes) == one_launch_pays(*runs, np.where(long > 1, 0, 1), np.full(B, left), *sizes)
    some = np.full(B, 1)                 # a slot whose sequence has ended early may have steps left: they do not count
    some[-1] = 0
    assert one_launch_pays(*runs, some, np.where(some > 0, left, 80000), *sizes) == one_launch_pays(*runs, some, some * left, *sizes)
