"""The decode step whose blocks run as thread-block clusters (decode_cluster.cu), against the general route of separate launches.

The general route is taken by a model one of whose matrices has no strip copy.  The cluster kernel takes every sum in the order of the general route's
kernels, so logits and residual stream are the same bit for bit (over more than 256 cached tokens, where it reads keys in another way, to rounding).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BASE = dict(num_layers=8, d_model=256, vocab_size=512, n_heads=4, n_kv_heads=4, mamba_d_state=16, mamba_expand=2, mamba_conv_kernel=4, mamba_head_dim=64,
            mamba_n_groups=1, attention_period=8, attention_slot=7)


def engines(cfg, rows, capacity):
    from reimagined_b200.decode import DecodeEngine, synthetic_params
    params = synthetic_params(cfg, seed=3, rope_positions=max(capacity, 16))
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
    """Sliding window shorter than the reply, positions that differ from what the cache holds, and a cache that runs full."""
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
