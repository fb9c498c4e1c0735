"""The decode step whose blocks run as thread-block clusters (decode_cluster.cu), against the general route of separate launches.

The general route is taken by a model one of whose matrices has no strip copy.  The cluster kernel takes every sum in the order of the general route's
kernels, so logits and residual stream are the same bit for bit (over more than 256 cached tokens, where it reads keys in another way, to rounding).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BASE = dict(num_layers=8, d_model=256, vocab_size=512, n_heads=4, n_kv_heads=4, mamba_d_state=16, mamba_expand=2, mamba_conv_kernel=4, mamba_head_dim=64,
            mamba_n_groups=1, attention_period=8, attention_slot=7)


def engines(cfg, rows, capacity, window=None, alone=False):
    """alone: a hybrid block adds its attention to the stream, and nothing else."""
    from reimagined_b200.decode import DecodeEngine, synthetic_params
    params = synthetic_params(cfg, seed=3, rope_positions=max(capacity, 16))
    for name in params:
        if window and name.endswith("attn.dims"):
            params[name][4] = window
        if alone and name.endswith(("mamba_gate", "attn_gate", "ffn_gate")):
            params[name][:] = name.endswith("attn_gate")
    clusters, general = (DecodeEngine(params, batch=rows, capacity=capacity) for _ in range(2))
    general._blocks[0].mamba.x.strips = None
    return params, clusters, general


@pytest.mark.parametrize("change,rows", [
    ({}, 1),                                                     # one sweep of the threads a row
    ({}, 8),                                                     # two sequences a cluster, the last cluster full
    ({}, 13),                                                    # the last cluster with one of two
    ({}, 64),                                                    # clusters of eight CTAs, the last one with four of five
    ({}, 121),                                                   # several waves
    (dict(n_heads=8, n_kv_heads=2), 3),                          # key/value heads shared by CTAs
    (dict(n_heads=16, n_kv_heads=16), 33),                       # 16-wide heads, as many as CTAs
    (dict(d_model=768, n_heads=6, n_kv_heads=6), 2),             # 128-wide heads, CTAs without any
    (dict(d_model=768, n_heads=12, n_kv_heads=12), 7),           # three weight blocks a strip
    (dict(d_model=512, n_heads=4, n_kv_heads=1, mamba_expand=3, mamba_head_dim=128), 40),
    (dict(d_model=1024, n_heads=16, n_kv_heads=16, num_layers=16), 1),
    (dict(d_model=2048, n_heads=32, n_kv_heads=32), 1),          # rows longer than one sweep
    (dict(num_layers=40), 2),                                    # more blocks than a launch takes
    (dict(attention_period=9), 5),                               # no attention at all
], ids=lambda v: "-".join(f"{k}{n}" for k, n in v.items()) if isinstance(v, dict) else str(v))
def test_blocks_in_clusters_match_separate_launches(cuda, tbl, change, rows):
    import gpu_helpers as H
    cfg = dict(BASE, **change)
    _, clusters, general = engines(cfg, rows, 8)
    rng = np.random.default_rng(rows)
    for t in range(4):
        ids = rng.integers(0, cfg["vocab_size"], rows).tolist()
        got, hidden = clusters.step(ids, trace=True)
        want, hidden_want = general.step(ids, trace=True)
        assert cuda.equal(hidden, hidden_want), f"token {t}: first block off {(hidden != hidden_want).flatten(1).any(dim=1).nonzero()[0]}"
        assert cuda.equal(got, want), f"token {t}"
    assert H.device_status() == 0
    assert clusters.capture() <= 6 < general.capture()


class Inner(int):
    """Stands where a configuration has the factor between model width and channels: any width gives this many."""

    def __mul__(self, width):
        return int(self)


@pytest.mark.parametrize("width,rows,in_clusters", [
    (3328, 1, True), (3328, 4, True),                            # as many parts of a row's sum of squares as the kernel adds: 8
    (3584, 1, False), (3584, 4, False), (4096, 2, False), (4352, 1, False), (4608, 3, False),      # more: separate launches
    (3584, 5, True),                                             # so many rows that the sum is taken in the other order, of any width
])
def test_residual_stream_wider_than_the_channels(cuda, tbl, width, rows, in_clusters):
    """A row's sum of squares is added up in the parts that the separate launches take it in, of which a wide row has more than the kernel has places for."""
    import gpu_helpers as H
    cfg = dict(BASE, d_model=width, mamba_expand=Inner(1024), num_layers=3, attention_period=9)
    _, clusters, general = engines(cfg, rows, 8)
    rng = np.random.default_rng(width)
    for t in range(3):
        ids = rng.integers(0, cfg["vocab_size"], rows).tolist()
        got, hidden = clusters.step(ids, trace=True)
        want, hidden_want = general.step(ids, trace=True)
        assert cuda.equal(hidden, hidden_want), f"token {t}: first block off {(hidden != hidden_want).flatten(1).any(dim=1).nonzero()[0]}"
        assert cuda.equal(got, want), f"token {t}"
    assert H.device_status() == 0
    assert (clusters.capture() <= 5) == in_clusters


@pytest.mark.parametrize("inner,taken", [(16384, True), (16640, False)])
def test_more_channels_than_a_step_takes(cuda, tbl, inner, taken):
    """Refused by either route."""
    import gpu_helpers as H
    cfg = dict(BASE, mamba_expand=Inner(inner), num_layers=1, attention_period=9)
    _, clusters, general = engines(cfg, 1, 8)
    for engine in (clusters, general):
        if taken:
            engine.step([5])
        else:
            with pytest.raises(Exception, match="tbl_decode_step"):
                engine.step([5])
    assert H.device_status() == 0 and (not taken or cuda.equal(clusters.logits, general.logits))


def filled(engine, seed, positions):
    """Every cache and state of the engine random, the sequences at the given positions."""
    import torch
    numbers = engine.state.view(torch.float32)
    numbers.copy_(torch.randn(numbers.shape, generator=torch.Generator("cuda").manual_seed(seed), device="cuda") * 2)
    numbers[:engine.batch].view(torch.int32).copy_(torch.as_tensor(positions, dtype=torch.int32))


# several sequences a cluster: 3, 5 and 8 of them, by 4, 2 and 1 warps a sequence's head
SEVERAL = [
    ({}, 16),
    ({}, 33),
    (dict(d_model=768, n_heads=16, n_kv_heads=16), 20),          # 48-wide heads, rows that do not divide the threads
    (dict(n_heads=2, n_kv_heads=1), 64),                         # 128-wide heads in clusters of eight CTAs
    (dict(n_heads=16, n_kv_heads=4), 50),                        # 16-wide heads, keys shared by CTAs
    (dict(d_model=768, n_heads=12, n_kv_heads=12), 56),          # no room for all partial sums of the values: eight rounds
]
IDS = [f"{'-'.join(f'{k}{n}' for k, n in c.items()) or 'base'}-{rows}" for c, rows in SEVERAL]


@pytest.mark.parametrize("window", [4096, 70])
@pytest.mark.parametrize("change,rows", SEVERAL, ids=IDS)
def test_attention_of_several_sequences_a_cluster(cuda, tbl, change, rows, window):
    """Up to 256 cached tokens, another number in every sequence: bit for bit, over more tokens than a sequence has threads."""
    import gpu_helpers as H
    cfg = dict(BASE, **change)
    params, clusters, general = engines(cfg, rows, 260, window)
    rng = np.random.default_rng(rows)
    positions = np.concatenate([[0, 1, 31, 32, 63, 64, 127, 128, 250], rng.integers(100, 252, rows)])[:rows]
    filled(clusters, rows, positions)
    general.state.copy_(clusters.state)
    for t in range(4):
        ids = rng.integers(0, cfg["vocab_size"], rows).tolist()
        got, hidden = clusters.step(ids, trace=True)
        want, hidden_want = general.step(ids, trace=True)
        assert cuda.equal(hidden, hidden_want), f"token {t}: first block off {(hidden != hidden_want).flatten(1).any(dim=1).nonzero()[0]}"
        assert cuda.equal(got, want), f"token {t}"
    assert H.device_status() == 0
    assert clusters.capture() <= 6 < general.capture()


@pytest.mark.parametrize("change,rows,tokens,window", [({}, 3, 900, 4096), *[(c, rows, 400 if rows == 56 else 700, 4096) for c, rows in SEVERAL],
                                                       ({}, 16, 900, 300), ({}, 33, 900, 257)], ids=lambda v: str(v) if isinstance(v, int) else "")
def test_attention_over_a_long_context(cuda, tbl, change, rows, tokens, window):
    """257 cached tokens and more: one step from the same random caches, what a hybrid block adds to the stream for its attention alone.  The two routes'
    results differ in the last places before the output projection takes them as 8-bit codes (3e-7 of a row's largest value, 4e-5 of a code's step), so
    that about one row in thirty has a value whose code moves: by one unit, of the some 500 that a sum of 256 such products comes to -- 2e-3 a code.
    A token left out or taken twice would be one part in the root of the tokens' number, 3e-2 to 6e-2, and a wrong key no less than 5e-3, in every row."""
    import gpu_helpers as H
    cfg = dict(BASE, attention_slot=0, **change)
    params, clusters, general = engines(cfg, rows, tokens, window, alone=True)
    positions = np.concatenate([[256, 257, 258, 287, 288, 319, 320, tokens - 3], np.random.default_rng(rows).integers(256, tokens - 2, rows)])[:rows]
    clean = []
    for seed in range(3):
        filled(clusters, seed, positions)
        general.state.copy_(clusters.state)
        ids = np.random.default_rng(seed).integers(0, cfg["vocab_size"], rows).tolist()
        got, want = ((h[1] - h[0]).double() for _, h in (e.step(ids, trace=True) for e in (clusters, general)))
        err = (got - want).abs().amax(dim=1) / want.abs().amax(dim=1)
        assert float(err.max()) <= 6e-3, f"sequence {int(err.argmax())}: {float(err.max())}"
        clean += (err <= 1e-5).tolist()
    assert np.mean(clean) >= 0.8, np.mean(clean)
    assert H.device_status() == 0
    assert clusters.capture() <= 6 < general.capture()


@pytest.mark.parametrize("change,rows", [SEVERAL[1], SEVERAL[3], ({}, 3)], ids=["base-33", "n_heads2-n_kv_heads1-64", "base-3"])
def test_value_sums_over_a_long_context(cuda, tbl, change, rows):
    """The weighted sum of the values adds hundreds of terms in 32 bits; it errs no more than the separate launches' sums.  All values are 1, so that the
    sum is 1 and all its 8-bit codes are 127: the output is the largest sum times a whole number, and shows its last places."""
    import gpu_helpers as H
    from reimagined_b200.decode import DecodeEngine, synthetic_params
    cfg = dict(BASE, attention_slot=0, **change)
    params = synthetic_params(cfg, seed=3)
    kv_dim = cfg["n_kv_heads"] * cfg["d_model"] // cfg["n_heads"]
    params["embedding"][:] = 0
    params["L0.mamba_gate"][:], params["L0.attn_gate"][:], params["L0.ffn_gate"][:] = 0, 1, 0
    params["L0.attn.kv.bias"][kv_dim:], params["L0.attn.out.bias"][:] = 1, 0
    words = params["L0.attn.out.words"].reshape(-1, 1) >> (2 * np.arange(16, dtype=np.uint32)) & 3
    sums = (words.reshape(cfg["d_model"], -1).astype(np.int64) - 1).sum(axis=1)
    column = int(np.abs(sums).argmax())
    exact = sums[column] * float(params["L0.attn.out.scale"][0])
    clusters, general = (DecodeEngine(params, batch=rows, capacity=704) for _ in range(2))
    general._blocks[0].mamba.x.strips = None
    errs = []
    for engine in (clusters, general):
        rng, err = np.random.default_rng(rows), []
        for _ in range(3 if rows > 3 else 30):
            engine.state.view(cuda.float32).fill_(1.0)
            engine.state[:4 * rows].view(cuda.int32).copy_(cuda.as_tensor(rng.integers(256, 700, rows), dtype=cuda.int32))
            _, hidden = engine.step([0] * rows, trace=True)
            err.append(hidden[1, :, column].double().cpu().numpy() / exact - 1)
        errs.append(float(np.sqrt(np.mean(np.square(err)))))
    assert errs[0] <= errs[1] <= 1e-6, errs
    assert H.device_status() == 0
    assert clusters.capture() <= 6 < general.capture()


@pytest.mark.parametrize("change,rows,short,beyond", [
    (dict(num_layers=1, attention_period=1, attention_slot=0), 64, 250, 300),          # every block attends
    ({}, 64, 2100, 2300),                                        # one block of eight
    (dict(n_heads=2, n_kv_heads=1), 64, 700, 800),               # heads twice as wide
    ({}, 1, 4000, None),                                         # one sequence: nowhere
])
def test_route_by_the_context(cuda, tbl, change, rows, short, beyond):
    """Clusters where they are faster over as many tokens as the cache takes, or the window lets a step see; either way the same logits."""
    import gpu_helpers as H
    cfg = dict(BASE, **change)
    for capacity, window, in_clusters in [(short, 4096, True), *([(beyond, 4096, False), (beyond, short, True), (short, beyond, True)] if beyond else [])]:
        _, clusters, general = engines(cfg, rows, capacity, window)
        ids = np.random.default_rng(rows).integers(0, cfg["vocab_size"], rows).tolist()
        for _ in range(2):
            assert cuda.equal(clusters.step(ids), general.step(ids)), (capacity, window)
        assert (clusters.capture() <= 6) == in_clusters, (capacity, window)
    assert H.device_status() == 0


def test_long_context_matches_separate_launches_to_rounding(cuda, tbl):
    """300 cached tokens: keys read by four lanes a token.  Scores in another order of sums, 1e-6 of their size, now and then move an 8-bit code by a
    step: 1 / 127 of the row's largest value in one of 256 terms of a sum, from which the rows drift; most steps agree far more closely."""
    import gpu_helpers as H
    _, clusters, general = engines(BASE, 3, 304)
    rng = np.random.default_rng(5)
    close = 0
    for t in range(300):
        ids = rng.integers(0, BASE["vocab_size"], 3).tolist()
        got, want = clusters.step(ids), general.step(ids)
        if t < 256:
            assert cuda.equal(got, want), t
        else:
            err = float((got - want).abs().max() / want.abs().max())
            assert err <= 1e-1, t
            close += err <= 1e-5
    assert close >= 1 and H.device_status() == 0


def test_clusters_match_the_oracle_through_a_long_window(cuda, port, tbl):
    """Sliding window shorter than the reply, and a cache that runs full."""
    import gpu_helpers as H
    from oracle.decode import PortDecoder
    cfg = dict(BASE)
    params, clusters, _ = engines(cfg, 2, 40)
    for name in [k for k in params if k.endswith("attn.dims")]:
        params[name][4] = 24
    from reimagined_b200.decode import DecodeEngine
    clusters = DecodeEngine(params, batch=2, capacity=40)
    oracle = PortDecoder(params, rows=2, capacity=40)
    rng = np.random.default_rng(8)
    close = 0
    for t in range(40):
        ids = rng.integers(0, cfg["vocab_size"], 2).tolist()
        got = clusters.step(ids).cpu().numpy()
        _, want = oracle.step(ids)
        err = np.abs(got - want).max() / np.abs(want).max()
        assert err <= 1e-1, t
        close += err <= 1e-3
    assert close >= 1 and H.device_status() == 0
    clusters.step(ids)                       # the cache is full: reported, and the step still ends
    assert H.device_status() == 4
