"""The register-resident forward kernel takes two batch rows per instruction.  Every operation must round on
its own, as in the shared-memory kernel, which takes one row at a time: the two then differ only where the
order of the synaptic sums does, in a small share of the voltages.  A contracted multiply-add changes a
third of them in the last bit."""
import dataclasses

import pytest
import torch


@pytest.mark.gpu
@pytest.mark.parametrize("batch,n_bkg", [(1, 20), (2, 20), (3, 20), (5, 20), (6, 20), (7, 20), (8, 20),
                                         (6, 200)])      # more counts per step than 2 per thread
@pytest.mark.parametrize("n_receptors", [4, 5])
def test_paired_rows_round_like_single_rows(batch, n_bkg, n_receptors):
    from util import make_case, make_inputs
    from v1_glif_model_b200 import synth
    from v1_glif_model_b200.models import V1Column
    cfg, dicts, _ = make_case(dataclasses.replace(synth.CONFIGS["small"], batch=batch, n_bkg=n_bkg, n_receptors=n_receptors))
    cell = V1Column(*dicts)
    x, c = (torch.from_numpy(t).cuda() for t in make_inputs(cfg, seq_len=40))
    out = []
    for smem in (0, 1):
        cell.set_option("force_smem_kernel", smem)
        z, v = cell.rollout(x, c)
        cell.synchronize()
        out.append((z, v, cell.counters()))
    (z1, v1, n1), (z2, v2, n2) = out
    assert int(z1.sum()) > 0 and torch.equal(z1, z2) and n1 == n2
    assert float((v1 != v2).float().mean()) < 0.01
