"""Forest-cascade decode attention (shared header / prompt nodes on tensor-core tiles + per-sequence pass + merge)
against a dense fp32 oracle, and the rollout engine's prefix-tree discovery end to end."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

PAGE = 16


def _scratch(B, Hq, D, splits):
    f32 = dict(device="cuda", dtype=torch.float32)
    return ([torch.empty((B, Hq, splits, D), **f32) for _ in range(4)],
            [torch.empty((B, Hq, splits, 2), **f32) for _ in range(4)])


def _forms(B, Hkv):
    """The op as three launches and as one, with the counters that the latter wants."""
    from arctic_platform_b200.ops import forest_attention as fa
    arrived = torch.zeros(2 * B * Hkv, device="cuda", dtype=torch.int32)
    return {"three": fa.forest_decode_attention_passes,
            "one": lambda *a, **k: fa.forest_decode_attention(*a, arrived=arrived, **k)}


@pytest.mark.parametrize("form", ["three", "one"])
@pytest.mark.parametrize("Hq,Hkv", [(32, 8), (32, 4), (16, 8)])
def test_shared_pass_when_single_rows_meet_much_larger_scores_late(form, Hq, Hkv):
    """The running reference of a row moves when its scores outgrow it by 2^8; here some rows of a warp do, others never, in
    several blocks.  bf16 weights and outputs (2^-8 at most each, half of that in the
    mean) against fp32."""
    from arctic_platform_b200.ops import _lib
    from arctic_platform_b200.ops import forest_attention as fa
    B, D, tokens = 12, 128, 1216
    g = torch.Generator(device="cuda").manual_seed(5)
    n = tokens // PAGE
    kc, vc = (torch.randn((n + B, Hkv, PAGE, D), generator=g, device="cuda").to(torch.bfloat16) for _ in range(2))
    q = torch.randn((B, Hq, D), generator=g, device="cuda")
    q[::3] *= 6                                    # scores of every third sequence spread six times as far ...
    kc[3 * n // 8:3 * n // 8 + 2] *= 3             # ... and grow in two of the ten blocks
    kc[7 * n // 8:7 * n // 8 + 1] *= 5
    q = q.to(torch.bfloat16)
    pages = np.arange(n, dtype=np.int32)
    own = [np.array([n + b], dtype=np.int32) for b in range(B)]
    forest = fa.build_forest_tables([fa.ForestNode(0, list(range(B)), pages, tokens)], B, n + 1, 128 * Hkv // Hq, "cuda")
    i32 = dict(device="cuda", dtype=torch.int32)
    table = torch.zeros((B, n + 1), **i32)
    table[:, 0] = torch.arange(n, n + B, **i32)
    part_o, part_ml = _scratch(B, Hq, D, 2)
    out = _forms(B, Hkv)[form](q, kc, vc, forest, torch.arange(B, **i32), torch.ones(B, **i32), table, torch.full((B,), 5, **i32), part_o,
                               part_ml, 2, 2)
    _lib.check_status("forest")
    ref = fa.forest_decode_reference(q, kc, vc, [[(pages, tokens), (own[b], 5)] for b in range(B)])
    assert (out.float() - ref).norm() <= 2 ** -7 * ref.norm()


@pytest.mark.parametrize("form", ["three", "one"])
@pytest.mark.parametrize("Hq,Hkv", [(32, 8), (16, 8), (8, 8), (32, 4), (16, 1)])
def test_three_level_forest_matches_dense_attention(Hq, Hkv, form):
    """Headers shared by several prompts, prompts shared by their rollouts, private tails; one sequence without a
    header, one prompt node whose slots are not consecutive, and a header with more sequences than one tile holds."""
    from arctic_platform_b200.ops import _lib
    from arctic_platform_b200.ops import forest_attention as fa
    D, splits = 128, 4
    R = Hq // Hkv
    max_rows = 128 // R
    B = max_rows + 12                      # the first header spans more sequences than one tile
    g = torch.Generator(device="cuda").manual_seed(3)
    num_pages = 400
    kc = torch.randn((num_pages, Hkv, PAGE, D), generator=g, device="cuda").to(torch.bfloat16)
    vc = torch.randn((num_pages, Hkv, PAGE, D), generator=g, device="cuda").to(torch.bfloat16)
    q = torch.randn((B, Hq, D), generator=g, device="cuda").to(torch.bfloat16)
    rng = np.random.default_rng(0)
    perm = rng.permutation(num_pages).astype(np.int32)
    nxt = [0]

    def take(n):
        out = perm[nxt[0]:nxt[0] + n]
        nxt[0] += n
        return out

    nodes, ctx = [], [[] for _ in range(B)]
    hdr_a, hdr_b = take(9), take(5)                                       # 144 and 80 tokens
    slots_a = list(range(0, max_rows + 4))
    slots_b = list(range(max_rows + 4, B - 1))                            # the last slot has no header at all
    nodes.append(fa.ForestNode(0, slots_a, hdr_a, 144))
    nodes.append(fa.ForestNode(0, slots_b, hdr_b, 80))
    for s in slots_a:
        ctx[s].append((hdr_a, 144))
    for s in slots_b:
        ctx[s].append((hdr_b, 80))
    # prompt nodes: groups of 4 slots; one group deliberately scattered
    groups = [list(range(i, min(i + 4, B))) for i in range(0, B, 4)]
    groups[1], groups[2] = [4, 5, 8, 9], [6, 7, 10, 11]
    for grp in groups:
        n_tok = int(rng.integers(1, 6)) * PAGE
        pg = take(n_tok // PAGE)
        nodes.append(fa.ForestNode(1, grp, pg, n_tok))
        for s in grp:
            ctx[s].append((pg, n_tok))
    max_pages = 16
    priv = np.zeros((B, max_pages), dtype=np.int32)
    plen = np.zeros(B, dtype=np.int32)
    for s in range(B):
        n = int(rng.integers(1, 40))
        pg = take((n + PAGE - 1) // PAGE)
        priv[s, :len(pg)] = pg
        plen[s] = n
        ctx[s].append((pg, n))
    forest = fa.build_forest_tables(nodes, B, max_pages, max_rows, "cuda")
    assert forest.n_levels == 2 and forest.n_nodes >= len(nodes) + 2       # scattered / oversized nodes take extra rows
    i32 = dict(device="cuda", dtype=torch.int32)
    po, pml = _scratch(B, Hq, D, splits)
    for buf in po + pml:
        buf.fill_(float("nan"))                                            # stale partials must never be merged
    out = _forms(B, Hkv)[form](q, kc, vc, forest, torch.arange(B, **i32), torch.ones(B, **i32), torch.from_numpy(priv).cuda(),
                               torch.from_numpy(plen).cuda(), po, pml, splits, 1)
    _lib.check_status("forest")
    ref = fa.forest_decode_reference(q, kc, vc, ctx)
    assert torch.isfinite(out.float()).all()
    assert (out.float() - ref).abs().max().item() < 2e-2


@pytest.mark.parametrize("Hq,Hkv,chunk,parts", [(32, 8, 4, 64), (32, 4, 16, 8), (16, 1, 1, 3), (8, 8, 2, 1)])
def test_own_pages_in_parts_with_and_without_shared_nodes(Hq, Hkv, chunk, parts):
    """Lengths at the edges of pages and parts, from nothing to more parts than allowed, an inactive entry; the same sequences once by
    themselves and once below a node that all but one share, whose parts outnumber its blocks.  bf16 probabilities and outputs (2^-9
    of a value each) against fp32; rows with nothing to see are zeros."""
    from arctic_platform_b200.ops import _lib
    from arctic_platform_b200.ops import forest_attention as fa
    D = 128
    lens = [0, 1, 15, 16, 17, 16 * chunk, 16 * chunk + 1, 16 * chunk * 2 + 5, 777, 1040, 300, 33]
    B, dead = len(lens), 9
    rows = min(B - 1, 128 // (Hq // Hkv))
    g = torch.Generator(device="cuda").manual_seed(Hq + chunk)
    max_pages, node_pages = 66, 20
    kc, vc = (torch.randn((B * max_pages + node_pages, Hkv, PAGE, D), generator=g, device="cuda").bfloat16() for _ in range(2))
    q = torch.randn((B, Hq, D), generator=g, device="cuda").bfloat16()
    perm = torch.randperm(B * max_pages, generator=g, device="cuda").to(torch.int32)
    table = perm.view(B, max_pages).contiguous()
    node = np.arange(B * max_pages, B * max_pages + node_pages, dtype=np.int32)
    i32 = dict(device="cuda", dtype=torch.int32)
    active = torch.ones(B, **i32)
    active[dead] = 0
    arrived = torch.zeros(2 * B * Hkv, **i32)
    for nodes in ([], [fa.ForestNode(0, list(range(rows)), node, node_pages * PAGE - 3)]):
        forest = fa.build_forest_tables(nodes, B, max_pages, 128 // (Hq // Hkv), "cuda")
        splits = 9
        part_o = [torch.full((B, Hq, n, D), float("nan"), device="cuda") for n in (splits, parts)]
        part_ml = [torch.full((B, Hq, n, 2), float("nan"), device="cuda") for n in (splits, parts)]
        own = torch.tensor(lens, **i32)
        for _ in range(2):                 # the second time from the counters that the first has left
            out = fa.forest_decode_attention(q, kc, vc, forest, torch.arange(B, **i32), active, table, own, part_o, part_ml, splits,
                                             parts, arrived=arrived, own_chunk=chunk)
        _lib.check_status("decode attention")
        assert not arrived.any()
        shared = [(node, node_pages * PAGE - 3)]
        ctx = [(shared if nodes and b < rows else []) + ([(table[b].cpu().numpy()[:(n + 15) // 16], n)] if b != dead else [])
               for b, n in enumerate(lens)]
        ref = fa.forest_decode_reference(q, kc, vc, ctx)
        assert torch.isfinite(out.float()).all()
        err = (out.float() - ref).norm(dim=-1)
        assert (err <= 2 ** -7 * ref.norm(dim=-1)).all()


@pytest.mark.parametrize("what", ["no mask", "many parts", "many own parts", "idle entries"])
def test_calls_that_the_one_launch_form_does_not_take(what):
    """Without a mask every source counts, parts may be more than 255, and what ``priv_start`` says of entries that are not live does
    not matter: such calls have the results of the three launches, with counters and without (entries that are not live: without).
    bf16 probabilities and outputs (2^-9 of a value each) against fp32."""
    from arctic_platform_b200.ops import _lib
    from arctic_platform_b200.ops import forest_attention as fa
    B, Hq, Hkv, D, pages = 6, 8, 2, 128, 5
    g = torch.Generator(device="cuda").manual_seed(len(what))
    kc, vc = (torch.randn((B * pages + 9, Hkv, PAGE, D), generator=g, device="cuda").bfloat16() for _ in range(2))
    q = torch.randn((B, Hq, D), generator=g, device="cuda").bfloat16()
    i32 = dict(device="cuda", dtype=torch.int32)
    table = torch.arange(B * pages, **i32).view(B, pages)
    node = np.arange(B * pages, B * pages + 9, dtype=np.int32)
    own = torch.tensor([70, 1, 80, 33, 16, 5], **i32)
    forest = fa.build_forest_tables([fa.ForestNode(0, list(range(B)), node, 140)], B, 9, 32, "cuda")
    start, active = torch.arange(B, **i32), torch.ones(B, **i32)
    splits = parts = 2
    live = list(range(B))
    if what == "no mask":
        forest.row_mask = None
    elif what == "many parts":
        splits = 300
    elif what == "many own parts":
        parts = 256
    else:
        active[1::2] = 0
        start[1], start[3], start[5] = 0, -1, 1 << 20
        live = [0, 2, 4]
    part_o = [torch.full((B, Hq, n, D), float("nan"), device="cuda") for n in (splits, parts)]
    part_ml = [torch.full((B, Hq, n, 2), float("nan"), device="cuda") for n in (splits, parts)]
    ref = fa.forest_decode_reference(q, kc, vc, [[(node, 140), (table[b].cpu().numpy()[:(n + 15) // 16], n)]
                                                for b, n in enumerate(own.tolist())])
    for arrived in [None] + ([] if what == "idle entries" else [torch.zeros(2 * B * Hkv, **i32)]):
        out = fa.forest_decode_attention(q, kc, vc, forest, start, active, table, own, part_o, part_ml, splits, parts, arrived=arrived)
        _lib.check_status("decode attention")
        err = (out[live].float() - ref[live]).norm(dim=-1)
        assert (err <= 2 ** -7 * ref[live].norm(dim=-1)).all()


@pytest.mark.parametrize("what", ["rows", "batch", "start", "own row", "idle row"])
def test_tables_beyond_the_tile_or_the_batch_are_reported(what):
    """One launch: more sequences than a tile has rows, sequences behind the batch, own rows outside of it.  What does not fit is
    left out, the status word says so, and with tables that hold and cleared counters the next call is right."""
    from arctic_platform_b200.ops import _lib
    from arctic_platform_b200.ops import forest_attention as fa
    B, Hq, Hkv, D, pages = 40, 16, 4, 128, 2
    g = torch.Generator(device="cuda").manual_seed(9)
    kc, vc = (torch.randn((B * pages + 9, Hkv, PAGE, D), generator=g, device="cuda").bfloat16() for _ in range(2))
    q = torch.randn((B, Hq, D), generator=g, device="cuda").bfloat16()
    i32 = dict(device="cuda", dtype=torch.int32)
    table = torch.arange(B * pages, **i32).view(B, pages)
    node = np.arange(B * pages, B * pages + 9, dtype=np.int32)
    own = torch.arange(B, **i32) % 32 + 1
    arrived = torch.zeros(2 * B * Hkv, **i32)
    part_o, part_ml = _scratch(B, Hq, D, 2)
    for wrong in (True, False):
        forest = fa.build_forest_tables([fa.ForestNode(0, list(range(B)), node, 140)], B, 9, 64 if wrong and what == "rows" else 32, "cuda")
        start, active = torch.arange(B, **i32), torch.ones(B, **i32)
        if wrong and what == "batch":
            forest.q_count[1] += 3
        elif wrong and what == "start":
            forest.q_start[1] = -8
        elif wrong and what == "own row":
            start[7] = B
        elif wrong and what == "idle row":
            start[7], active[7] = -1, 0
        out = fa.forest_decode_attention(q, kc, vc, forest, start, active, table, own, part_o, part_ml, 2, 2, arrived=arrived)
        if wrong:
            with pytest.raises(_lib.KernelError, match="203"):
                _lib.check_status("decode attention")
            arrived.zero_()
    _lib.check_status("decode attention")
    ref = fa.forest_decode_reference(q, kc, vc, [[(node, 140), (table[b].cpu().numpy()[:(n + 15) // 16], n)]
                                                for b, n in enumerate(own.tolist())])
    err = (out.float() - ref).norm(dim=-1)
    assert (err <= 2 ** -7 * ref.norm(dim=-1)).all()


def test_engine_discovers_shared_headers_and_samples_the_same_distribution():
    """Prompts that start with the same tokens are stored and attended through one header node.  Greedy generation with
    the forest equals greedy generation with plain per-sequence decoding, and the reported log-probs match a
    teacher-forced scoring pass."""
    from arctic_platform_b200.engine.sampler import SamplerEngine
    from arctic_platform_b200.models.config import PRESETS
    from arctic_platform_b200.models.decoder import DecoderLM
    from arctic_platform_b200.ops import _lib
    cfg = PRESETS["qwen3-tiny-d128"]
    model = DecoderLM(cfg, "cuda", torch.bfloat16).init_weights(seed=5)
    g = torch.Generator().manual_seed(1)
    header = torch.randint(1, cfg.vocab_size, (100,), generator=g).tolist()      # 6 full pages in common
    prompts = [header + torch.randint(1, cfg.vocab_size, (n,), generator=g).tolist() for n in (21, 40, 7)]
    prompts.append(torch.randint(1, cfg.vocab_size, (57,), generator=g).tolist())  # shares nothing
    sp = {"n": 3, "temperature": 0.0, "max_tokens": 12, "ignore_eos": True}
    outs = {}
    for cascade in (True, False):
        eng = SamplerEngine(cfg, "cuda", model=model, kv_cache_tokens=1 << 14, max_batch=16, max_seq_len=512,
                            cascade=cascade, use_cuda_graph=False)
        if cascade:
            runs = eng._plan_runs([np.asarray(p, dtype=np.int64) for p in prompts])
            assert sorted(map(tuple, (r[0] for r in runs))) == [(0, 1, 2), (3,)]
            assert dict((tuple(r[0]), r[1]) for r in runs)[(0, 1, 2)] == 96      # page-aligned part of the 100 tokens
        outs[cascade] = eng.generate(prompts, sp)
        if cascade:
            assert eng.n_levels == 2 and eng.forest_stats["shared_tokens"] > 0
        _lib.check_status("forest engine")
    for a, b in zip(outs[True], outs[False]):
        assert a["prompt_index"] == b["prompt_index"] and a["token_ids"] == b["token_ids"]
        assert a["logprobs"] == pytest.approx(b["logprobs"], abs=5e-2)


@pytest.mark.parametrize("switch", ["none", "splits", "scalar"])
def test_switches_of_the_per_sequence_pass_reach_models_that_share_a_prompt(switch, monkeypatch):
    """``APB_DECODE_SEQ_SPLITS`` and the scalar kernel belong to the three launches, so with either of them a rollout makes these; the
    tokens are those of the one launch, log-probabilities agree to the roundings of bf16 probabilities."""
    from arctic_platform_b200.engine import sampler
    from arctic_platform_b200.models.config import PRESETS
    from arctic_platform_b200.models.decoder import DecoderLM
    from arctic_platform_b200.ops import _lib
    cfg = PRESETS["qwen3-tiny-d128"]
    model = DecoderLM(cfg, "cuda", torch.bfloat16).init_weights(seed=5)
    prompt = torch.randint(1, cfg.vocab_size, (70,), generator=torch.Generator().manual_seed(2)).tolist()
    eng = sampler.SamplerEngine(cfg, "cuda", model=model, kv_cache_tokens=1 << 12, max_batch=8, max_seq_len=128, use_cuda_graph=False)
    sp = {"n": 4, "temperature": 0.0, "max_tokens": 6, "ignore_eos": True}
    plain = eng.generate([prompt], sp)
    seen = []
    for name in ("forest_decode_attention", "forest_decode_attention_passes"):
        monkeypatch.setattr(sampler, name, lambda *a, _f=getattr(sampler, name), _n=name, **k: seen.append((_n, a[11])) or _f(*a, **k))
    if switch == "splits":
        monkeypatch.setenv("APB_DECODE_SEQ_SPLITS", "3")
    _lib.cuda_lib().apb_decode_use_scalar(int(switch == "scalar"))
    try:
        out = eng.generate([prompt], sp)
    finally:
        _lib.cuda_lib().apb_decode_use_scalar(0)
    _lib.check_status("switches")
    assert {n for n, _ in seen} == {"forest_decode_attention" if switch == "none" else "forest_decode_attention_passes"}
    if switch == "splits":
        assert {s for _, s in seen} == {3}
    for a, b in zip(out, plain):
        assert a["token_ids"] == b["token_ids"] and a["logprobs"] == pytest.approx(b["logprobs"], abs=5e-2)


def test_rollout_chooses_a_form_when_sequences_join(monkeypatch):
    """Rollouts that keep to either form, or take one and then the other as prompts join (4 slots, so the second prompt waits for the
    first), have the same tokens, captured or not; the rule is asked when sequences have joined and told what is on the device."""
    from arctic_platform_b200.engine import sampler
    from arctic_platform_b200.models.config import PRESETS
    from arctic_platform_b200.models.decoder import DecoderLM
    from arctic_platform_b200.ops import _lib
    cfg = PRESETS["qwen3-tiny-d128"]
    model = DecoderLM(cfg, "cuda", torch.bfloat16).init_weights(seed=5)
    g = torch.Generator().manual_seed(3)
    prompts = [torch.randint(1, cfg.vocab_size, (n,), generator=g).tolist() for n in (70, 33)]
    sp = {"n": 3, "temperature": 0.0, "max_tokens": 40, "ignore_eos": True}
    outs = {}
    for name, rule in (("one", lambda own: True), ("three", lambda own: False), ("turns", lambda own: own[0] == 70 % PAGE + 1)):
        for graph in (False, True):
            told = []
            eng = sampler.SamplerEngine(cfg, "cuda", model=model, kv_cache_tokens=1 << 12, max_batch=4, max_seq_len=128, sync_interval=8,
                                        use_cuda_graph=graph)

            def pays(node_tokens, node_slots, own, left, *sizes, _r=rule):
                told.append((list(node_tokens), list(node_slots), list(own), list(left)))
                assert eng.d_priv_len[:len(own)].tolist() == told[-1][2]
                return _r(own)
            monkeypatch.setattr(sampler, "one_launch_pays", pays)
            outs[name, graph] = [eng.generate(prompts, sp) for _ in range(2)]
            assert len(eng._graphs) == (0 if not graph else 2 if name == "turns" else 1)
            want = [([64], [3], [70 % PAGE + 1] * 3 + [0], [39] * 3), ([32], [3], [33 % PAGE + 1] * 3 + [0], [39] * 3)]
            assert [(a, b, c, d[:3]) for a, b, c, d in told] == want * 2
        _lib.check_status("rollout")
    want = outs["one", False][0]
    for got in outs.values():
        for call in got:
            for a, b in zip(call, want):
                assert a["token_ids"] == b["token_ids"] and a["logprobs"] == pytest.approx(b["logprobs"], abs=5e-2)


def test_counters_that_a_failed_call_left_behind_do_not_reach_the_next_one():
    """A call that an error ends between launches may leave arrivals: the next call begins with counters of zero."""
    from arctic_platform_b200.engine import sampler
    from arctic_platform_b200.models.config import PRESETS
    from arctic_platform_b200.models.decoder import DecoderLM
    from arctic_platform_b200.ops import _lib
    cfg = PRESETS["qwen3-tiny-d128"]
    model = DecoderLM(cfg, "cuda", torch.bfloat16).init_weights(seed=5)
    prompt = torch.randint(1, cfg.vocab_size, (70,), generator=torch.Generator().manual_seed(2)).tolist()
    eng = sampler.SamplerEngine(cfg, "cuda", model=model, kv_cache_tokens=1 << 12, max_batch=8, max_seq_len=128)
    sp = {"n": 4, "temperature": 0.0, "max_tokens": 6, "ignore_eos": True}
    want = eng.generate([prompt], sp)
    assert eng._one_launch and not eng.d_arrived.any()
    eng.d_arrived.copy_(torch.arange(eng.d_arrived.numel()) % 5)          # as from a kernel that gave up
    got = eng.generate([prompt], sp)
    _lib.check_status("after arrivals")
    assert not eng.d_arrived.any()
    for a, b in zip(got, want):
        assert a["token_ids"] == b["token_ids"] and a["logprobs"] == pytest.approx(b["logprobs"], abs=5e-2)


@pytest.mark.parametrize("form", ["three", "one"])
@pytest.mark.parametrize("Hq,Hkv,samples,tokens", [(32, 8, 16, 2175), (32, 8, 8, 300), (32, 4, 16, 4000), (16, 2, 4, 1000)])
def test_repeats_have_the_same_bits_whatever_arrives_first(form, Hq, Hkv, samples, tokens):
    """Nodes whose pages come from memory late and in any order (caches of 180 MB in turn, more than the L2 holds): a product that is
    read before it has landed changes the result.  Parts are joined in the order of their places, so repeats are equal to the bit; and
    they are near fp32 (bf16 weights and outputs, 2^-9 of a value each)."""
    from arctic_platform_b200.ops import _lib
    from arctic_platform_b200.ops import forest_attention as fa
    D, n = 128, (tokens + PAGE - 1) // PAGE
    i32 = dict(device="cuda", dtype=torch.int32)
    g = torch.Generator(device="cuda").manual_seed(tokens)
    layers = -(-180_000_000 // (n * Hkv * PAGE * D * 4))
    kc, vc = (torch.randn((layers, n + samples, Hkv, PAGE, D), generator=g, device="cuda").bfloat16() for _ in range(2))
    q = torch.randn((samples, Hq, D), generator=g, device="cuda").bfloat16()
    pages = np.arange(n, dtype=np.int32)
    forest = fa.build_forest_tables([fa.ForestNode(0, list(range(samples)), pages, tokens)], samples, n, 128 * Hkv // Hq, "cuda")
    table = torch.arange(n, n + samples, **i32).view(-1, 1)
    splits = max(1, min(8, 148 // Hkv))
    part_o, part_ml = _scratch(samples, Hq, D, splits)
    run = _forms(samples, Hkv)[form]
    args = (forest, torch.arange(samples, **i32), torch.ones(samples, **i32), table, torch.full((samples,), 9, **i32), part_o, part_ml, splits, 4)
    first = [run(q, kc[i], vc[i], *args) for i in range(layers)]
    for _ in range(max(3, 600 // layers)):
        for i in range(layers):
            assert torch.equal(run(q, kc[i], vc[i], *args), first[i])
    _lib.check_status("forest")
    ref = fa.forest_decode_reference(q, kc[0], vc[0], [[(pages, tokens), (np.array([n + b]), 9)] for b in range(samples)])
    assert ((first[0].float() - ref).norm(dim=-1) <= 2 ** -7 * ref.norm(dim=-1)).all()
