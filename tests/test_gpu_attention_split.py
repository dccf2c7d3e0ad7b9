"""The tensor-core attention core with the keys of a query tile shared by a cluster (csrc/attention_tc.cu): two and four CTAs, parts
without a key tile (the first causal query tiles), ragged last tiles, and the sizes on either side of the rule that splits."""
import numpy as np
import pytest

from oracle import port

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rt():
    from mimir_framework_b200 import runtime

    runtime.init(0)
    return runtime


@pytest.mark.parametrize("causal", [0, 1])
@pytest.mark.parametrize("batch,seq,heads", [(1, 192, 2), (1, 193, 3), (2, 449, 1), (1, 513, 2), (1, 1000, 12), (18, 512, 1), (19, 512, 1), (37, 512, 1), (38, 512, 1)])
def test_split_keys_against_the_port(rt, batch, seq, heads, causal):
    r = np.random.default_rng(batch + seq + heads + causal)
    E = 64 * heads
    x = r.standard_normal(batch * seq * E).astype(np.float32)
    w = (r.standard_normal(4 * E * E) / np.sqrt(E)).astype(np.float32)
    got = np.asarray(rt.attention(x, w, batch, seq, E, heads, causal)).reshape(batch, -1)
    for i in sorted({0, batch // 2, batch - 1}):
        want = port.attention(x[i * seq * E:(i + 1) * seq * E], w, seq, E, heads, causal).ravel()
        assert np.linalg.norm(got[i] - want) <= 1e-5 * np.linalg.norm(want)
        assert np.abs(got[i] - want).max() <= 1e-4 * np.abs(want).max()


# 1 000 keys and 12 heads: two parts; 513: four; 19 x 512: two; 38 x 512 and 192 keys: one CTA for all keys of a query tile
@pytest.mark.parametrize("causal", [0, 1])
@pytest.mark.parametrize("batch,seq,heads", [(1, 1000, 12), (1, 513, 2), (19, 512, 1), (38, 512, 1), (1, 192, 2)])
@pytest.mark.parametrize("where", ["first", "last"])
def test_an_overflowing_row_stays_visible(rt, batch, seq, heads, causal, where):
    """Activations beyond the half planes' range: every row that sees the overflowed key is non-finite, whichever part its key is in."""
    r = np.random.default_rng(seq + causal)
    E = 64 * heads
    x = r.standard_normal((batch, seq, E)).astype(np.float32)
    w = (r.standard_normal(4 * E * E) / np.sqrt(E)).astype(np.float32)
    at = 3 if where == "first" else seq - 5
    x[batch - 1, at] *= 1e7
    got = np.asarray(rt.attention(x.ravel(), w, batch, seq, E, heads, causal)).reshape(batch, seq, E)
    assert not np.isfinite(got[batch - 1, at if causal else 0:]).any()
    assert np.isfinite(got[:batch - 1]).all()
