"""The result table on the GPU where the measurements are split into parts and
the pairs into tiles unevenly: fewer measurements than parts, a tile that is
not full, more tiles than a wave of blocks.  Against the host restatement; the
two add the same doubles in another order (at most 6000 of them, all of one
sign: 1e-12 relative), the errors come from differences of those."""
import importlib

import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("n_meas,ndis,nrep", [(1, 32, 4), (3, 37, 7), (130, 11, 24), (700, 3, 5), (2, 6400, 24)])
def test_table_of_uneven_parts(csg, tmp_path, n_meas, ndis, nrep):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    an = importlib.import_module("spin_glass_b200.analysis")
    rng = np.random.default_rng(n_meas + ndis)
    rec = np.zeros((2 * n_meas, ndis, nrep), an.OBS_DT)
    rec["e"] = rng.uniform(-1.7, -0.5, rec["e"].shape)
    rec["m"] = rng.uniform(0.1, 0.2, rec["m"].shape)
    rec["q_0"] = rng.normal(0, 0.6, rec["q_0"].shape)
    rec["q_1_r"] = rng.normal(0, 0.1, rec["q_1_r"].shape)
    rec["q_1_i"] = rng.normal(0, 0.1, rec["q_1_i"].shape)
    path = str(tmp_path / "obs.bin")
    rec.tofile(path)
    host, gpu = an.analyze(path, 8, ndis, nrep), an.analyze_gpu(path, 8, ndis, nrep)
    assert gpu["n_meas"] == host["n_meas"] == n_meas
    for k in ("chi0", "xi", "e", "m"):
        np.testing.assert_allclose(gpu[k], host[k], rtol=1e-11, err_msg=k)
    for k in ("chi0_err", "xi_err", "e_err", "m_err"):
        np.testing.assert_allclose(gpu[k], host[k], rtol=1e-9, err_msg=k)
