"""LGN event lists built from words of spike flags: rows of a multiple of 8 and of 4 bytes, odd rows, rows
over several segments, and an address that allows no words.  The rollout's event counters count the list,
and the voltages equal the rollout over the same spikes read byte by byte (sums in another order: 1e-5)."""
import dataclasses

import numpy as np
import pytest
import torch


@pytest.mark.gpu
@pytest.mark.parametrize("n_lgn", [8, 12, 13, 96, 4096, 4100, 8200, 12289])
def test_event_list_is_the_same_for_every_word_size(n_lgn):
    from util import make_case
    from v1_glif_model_b200 import synth
    from v1_glif_model_b200.models import V1Column
    cfg, dicts, _ = make_case(dataclasses.replace(synth.CONFIGS["small"], n_lgn=n_lgn))
    cell = V1Column(*dicts)
    rng = np.random.default_rng(n_lgn)
    b, t = 3, 25
    p = np.where(np.arange(t) % 5 == 0, 0.0, 0.02)[None, :, None]
    x = (rng.random((b, t, n_lgn)) < p).astype(np.uint8)
    x[0, 1, :] = 1                        # a full row, an empty one and the ends of a row
    x[1, 2, [0, -1]] = 255
    counts = torch.zeros((b, t, cfg.n_bkg), dtype=torch.int32, device="cuda")
    z, v = cell.rollout(torch.from_numpy(x).cuda(), counts)
    cell.synchronize()
    assert cell.counters()["lgn_rows"] == int((x > 0).sum())
    odd = torch.empty(x.size + 1, dtype=torch.uint8, device="cuda")[1:].view(b, t, n_lgn)
    odd.copy_(torch.from_numpy(x))
    assert odd.data_ptr() % 4 and odd.is_contiguous()
    z2, v2 = cell.rollout(odd, counts)
    cell.synchronize()
    assert cell.counters()["lgn_rows"] == int((x > 0).sum())
    assert float((v - v2).norm()) <= 1e-5 * float(v.norm())
