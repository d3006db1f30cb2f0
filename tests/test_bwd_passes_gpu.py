"""The backward sweep handles three steps per pass: rollout lengths around the pass boundaries, delay ranges
around the ring size, every layout of the ring rows."""
import dataclasses

import pytest
import torch

from util import assert_grad_close, cuda_loss_spec, make_cells, make_inputs, oracle_loss_and_grads, state_to_oracle
from v1_glif_model_b200 import synth

pytestmark = pytest.mark.gpu
KW = dict(dampening_factor=0.5, pseudo_width=0.5)
LOSS = dict(rate_cost=10.0, voltage_cost=1e-1, sync_cost=0.0)


@pytest.mark.parametrize("delay", [1, 4, 5, 8])
@pytest.mark.parametrize("batch,channels,dense,options", [
    (2, 5, False, ()), (5, 5, False, ()), (7, 4, False, ()), (3, 4, True, ()), (5, 4, True, ()), (6, 5, True, ()),
    (5, 4, False, (("no_meta", 1),)), (5, 5, True, (("no_meta", 1),)), (5, 5, False, (("rollout_chunk", 32),)),
    (5, 5, False, (("state_in_global", 1),))])
def test_gradients_at_the_pass_boundaries(batch, channels, dense, options, delay):
    net = dataclasses.replace(synth.CONFIGS["tiny"], max_delay=delay)
    cfg, dicts, orc, cell = make_cells(net, options=options, seed=3, dense_basis=dense, n_receptors=channels, **KW)
    vscale = orc.params["voltage_scale"][orc.params["node_type_ids"]]
    # a carried state with spikes pending, so that even one step has gradients of every kind
    x, c = make_inputs(cfg, batch, 24, seed=5)
    state = cell.zero_state(batch)
    cell.rollout(torch.from_numpy(x).cuda(), torch.from_numpy(c).cuda(), state=state)
    st_o = state_to_oracle(state)
    for steps in (1, 2, 3, 4, 5, 7, 11):
        x, c = make_inputs(cfg, batch, steps, seed=20 + steps)
        st = tuple(t.clone() for t in state)
        if steps < 3:       # a current reaches the membrane two steps later: nothing depends on the weights yet
            cell.rollout(torch.from_numpy(x).cuda(), torch.from_numpy(c).cuda(), state=st, save_for_bwd=True)
            got = cell.backward(cuda_loss_spec(cfg, cell, LOSS))
            cell.synchronize()
            assert all(float(g.abs().max()) == 0.0 for g in got[:3])
            continue
        z, v, total, want = oracle_loss_and_grads(orc, cfg, x, c, vscale, LOSS, state=st_o)
        zc, _ = cell.rollout(torch.from_numpy(x).cuda(), torch.from_numpy(c).cuda(), state=st, save_for_bwd=True)
        assert torch.equal(zc.cpu().float(), z)
        got = cell.backward(cuda_loss_spec(cfg, cell, LOSS))
        cell.synchronize()
        for g, w, name in zip(got[:3], want, ("rec", "lgn", "bkg")):
            assert_grad_close(g, w, f"T={steps} {name}")
