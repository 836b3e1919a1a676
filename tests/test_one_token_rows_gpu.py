"""One-token steps of bf16 decoder models: the row kernels that keep a row in a block's registers, at widths where a block's last
warp is partly or barely used, one and several sequences, and beyond their largest width."""
import numpy as np
import pytest

import decoder_models as dm
from oracle import budurax, lutelorn

pytestmark = pytest.mark.gpu

TOL = 3e-2      # of the logits' scale per row: bf16 models, the bound of the other decoder tests


@pytest.mark.parametrize("sequences", [1, 3])
@pytest.mark.parametrize("width", [8, 33, 128, 132, 1000, 4096, 4104])
@pytest.mark.parametrize("architecture", ["budurax", "lutelorn"])
def test_decoding_at_row_widths(tmp_path, architecture, width, sequences):
    if architecture == "budurax":
        c = dm.config([dm.mamba(heads=3, vdim=24, norm_groups=1, groups=1), dm.latent(), dm.mamba(ff=None)], width=width)
        w, forward = dm.weights(c, 5), budurax.forward
    else:
        c = dm.lutelorn([dm.lightning(), dm.wkv(), dm.attention()], width=width)
        w, forward = dm.lutelorn_weights(c, 5), lutelorn.forward
    model = dm.load(tmp_path, c, w, "bfloat16")
    tokens = np.random.default_rng(width).integers(0, c["vocab"], (sequences, 14))
    want = [forward(c, w, t) for t in tokens]
    seqs = [model.open(14) for _ in range(sequences)]
    got = [model.step([(q, t[:5]) for q, t in zip(seqs, tokens)], [5 * (i + 1) - 1 for i in range(sequences)])]
    for k in range(5, 14):
        got.append(model.step([(q, t[k:k + 1]) for q, t in zip(seqs, tokens)], range(sequences)))
    got = np.stack(got)
    for i in range(sequences):
        assert dm.close(got[:, i], want[i][4:], TOL), (architecture, width, i)
    model.close_model()
