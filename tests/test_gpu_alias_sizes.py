"""GPU: environment alias tables at the edges of the table kernel -- one texel, rows that are no multiple of a
warp, a row of zero weight, tables too long for shared memory -- each texel's implied probability within 1e-6
relative of the FP64 distribution (the bound of test_gpu_env_tables.py)."""
import numpy as np
import pytest

import volprim_b200 as vp
from test_gpu_env_tables import implied_texel_probability

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w, h", [(1, 1), (2, 1), (1, 33), (31, 4), (32, 3), (33, 5), (511, 255), (20000, 3), (3, 20000)])
def test_sizes(vp_ctx, w, h):
    rng = np.random.default_rng(w + 7 * h)
    rgb = np.exp(rng.normal(0.0, 1.5, (h, w, 3))).astype(np.float32)
    if h >= 4:
        rgb[2] = 0.0
    env = vp.Environment(vp_ctx, rgb=rgb)
    t = env.tables()
    env.close()
    lum = 0.2126 * rgb[..., 0].astype(np.float64) + 0.7152 * rgb[..., 1] + 0.0722 * rgb[..., 2]
    wt = lum * np.sin((np.arange(h) + 0.5) / h * np.pi)[:, None]
    p = implied_texel_probability(t["cond_prob"], t["cond_alias"], t["marg_prob"], t["marg_alias"])
    want = wt / wt.sum()
    assert t["cond_alias"].max() < w and t["marg_alias"].max() < h
    assert np.all(np.abs(p - want) <= 1e-6 * want)
