"""Operator-level currents and their gradients against plain float64 sums over the synapse lists, at the
sizes where the kernels change their split: batch rows padded to 1, 2, 4 and 8 and more than 8, few synapse
types and many, short rows (one delay of one neuron), and rows long enough to be shared by several warps.

Tolerance: float32 sums of n products differ from the exact sum by at most n * 2^-24 * sum|terms|, and far
less for signed terms; 2e-6 in relative 2-norm covers the longest row here (900 terms).
"""
import dataclasses

import numpy as np
import pytest
import torch

TOL = 2e-6


def rel(got, want):
    want = want.double()
    return float((got.double().cpu() - want).norm() / want.norm().clamp_min(1e-30))


@pytest.mark.gpu
@pytest.mark.parametrize("n_bkg", [20, 2])
@pytest.mark.parametrize("batch,dense", [(1, False), (2, True), (3, False), (5, False), (5, True), (8, True), (9, False), (1, True)])
def test_currents_and_gradients_match_sums_over_the_synapses(batch, dense, n_bkg):
    from util import make_case
    from v1_glif_model_b200 import _lib, synth
    from v1_glif_model_b200.models import V1Column
    cfg0 = dataclasses.replace(synth.CONFIGS["small"], n_bkg=n_bkg, bkg_in_degree=min(3, n_bkg), n_receptors=4 if dense else 5)
    cfg, dicts, _ = make_case(cfg0, dense_basis=dense)
    cell = V1Column(*dicts)
    rng = np.random.default_rng(batch)
    n, r = cfg.n_neurons, cell.synaptic_basis_weights.shape[1]
    basis = torch.from_numpy(cell.synaptic_basis_weights).double()
    sources = [(_lib.SRC_REC, cell.recurrent_indices, cell.recurrent_weight_values, dicts[0]["synapses"]["syn_ids"],
                cell.recurrent_dense_shape[1], 0.05),
               (_lib.SRC_LGN, cell.input_indices, cell.input_weight_values, dicts[1]["syn_ids"], cell.input_dim, 0.2),
               (_lib.SRC_BKG, cell.bkg_input_indices, cell.bkg_input_weights, dicts[2]["syn_ids"], cell.n_bkg, 0.6)]
    dy = torch.from_numpy(rng.normal(size=(batch * n, r)).astype(np.float32))
    for src, idx, w, sid, n_cols, p in sources:
        x = (rng.random((batch, n_cols)) < p).astype(np.float32)
        if src == _lib.SRC_BKG:
            x *= rng.integers(1, 4, x.shape)
        x[:, 0] = 1.0
        post, pre = torch.from_numpy(idx[:, 0].copy()), torch.from_numpy(idx[:, 1].copy())
        sid = torch.from_numpy(np.asarray(sid).astype(np.int64))
        xt, w64 = torch.from_numpy(x).double(), w.double().cpu()
        active = (xt[:, pre] > 0).double() * (xt[:, pre] if src == _lib.SRC_BKG else 1.0)        # [B, nnz]
        per = basis[sid]                                                                         # [nnz, R]
        cur = torch.zeros(batch, n, r, dtype=torch.float64)
        cur.index_add_(1, post, (active * w64)[..., None] * per)
        assert rel(cell._syn_currents(src, torch.from_numpy(x).cuda()), cur.reshape(batch * n, r)) <= TOL
        g = (dy.double().reshape(batch, n, r)[:, post] * per).sum(-1)                            # [B, nnz]
        d_x = torch.zeros(batch, n_cols, dtype=torch.float64)
        d_x.index_add_(1, pre, g * w64)
        got_x, got_w = cell.syn_currents_grad(src, torch.from_numpy(x).cuda(), dy.cuda())
        assert rel(got_x, d_x) <= TOL
        assert rel(got_w, (g * active).sum(0)) <= TOL
