"""The FP64 pipeline replayed as a CUDA graph gives the bits of its eager launches, with the inputs of the call."""
import numpy as np
import pytest

from oracle import gprat_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n, m, blocks", [(700, 90, None), (1409, 33, "2")])
def test_graph_replay(monkeypatch, n, m, blocks):
    import torch

    from gprat_b200 import capi

    if blocks:
        monkeypatch.setenv("GPRAT_CU_FP64_PANEL_BLOCKS", blocks)
    d, h1, h2 = 8, (1.0, 1.0, 0.1), (0.7, 1.3, 0.02)
    x, y, xt = O.synthetic(n, m, d)
    xt2 = np.random.default_rng(2).standard_normal(xt.size)
    dev = torch.device("cuda", 0)
    dxt = torch.empty(xt.size, dtype=torch.float64, device=dev)

    def outputs():
        return [torch.empty(m, dtype=torch.float64, device=dev) for _ in range(2)]

    def run(gp, h, series, out):
        dxt.copy_(torch.from_numpy(series))
        for o in out:
            o.fill_(np.nan)
        gp.fit_predict_device(h, dxt.data_ptr(), dxt.numel(), m, out[0].data_ptr(), out[1].data_ptr(),
                              torch.cuda.current_stream(dev).cuda_stream)
        torch.cuda.synchronize()
        gp.check_status()
        return [o.cpu().numpy().copy() for o in out]

    calls = [(h1, xt), (h1, xt), (h1, xt), (h2, xt), (h2, xt2), (h1, xt2), (h1, xt)]
    monkeypatch.setenv("GPRAT_CU_GRAPH", "0")
    gp = capi.CudaGP(x, y, 1, n, d)
    want = [run(gp, h, s, outputs()) for h, s in calls]
    gp.close()
    monkeypatch.setenv("GPRAT_CU_GRAPH", "1")
    gp = capi.CudaGP(x, y, 1, n, d)
    out = outputs()
    for (h, s), w in zip(calls, want):  # eager, captured, then replayed
        got = run(gp, h, s, out)
        assert np.array_equal(got[0], w[0]) and np.array_equal(got[1], w[1])
    other = outputs()  # other addresses: eager, captured, replayed again
    for _ in range(3):
        got = run(gp, h1, xt, other)
        assert np.array_equal(got[0], want[0][0]) and np.array_equal(got[1], want[0][1])
    om, ov = O.OracleGP(x, y, 1, n, d, h1).predict_with_uncertainty(xt, 1, m)
    assert np.max(np.abs(got[0] - om)) <= 1e-10 * np.max(np.abs(om))
    assert np.max(np.abs(got[1] - ov) / ov) <= 1e-10
    gp.close()
