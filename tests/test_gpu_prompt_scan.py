"""The DeltaNet scan of a prompt at the edges of its groups of eight rows and of its grid (a block per value head and 32 columns: one an SM
where they all fit, as many as there is room for beyond)."""
import numpy as np
import pytest
import torch

from helpers import rel_err
from test_gpu_ops import _gdn_inputs, dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nk,nv", [(2, 2), (16, 32), (20, 40)])
@pytest.mark.parametrize("T", [1, 7, 8, 9, 31, 33])
def test_scan_equals_the_windows_rows(F, T, nk, nv):
    hs, NS, cur = 128, 34, 3
    rng = np.random.default_rng(100 * T + nv)
    ch, qkvz, ab, convw, dt, a, nw = _gdn_inputs(rng, T, nk, nv, hs)
    S0, h0 = (0.1 * rng.standard_normal((NS, nv, hs, hs))).astype(np.float32), rng.standard_normal((NS, 3, ch)).astype(np.float32)
    args = (dev(convw), dev(dt), dev(a), dev(nw))
    W = min(T, 32)   # (a window's rows at most)
    Sw, Hw, Sp, Hp = dev(S0), dev(h0), dev(S0), dev(h0)
    want = [F.gdn_core(dev(qkvz[:W]), dev(ab[:W]), Hw, *args, Sw, dev(np.array([cur], np.int32)), None, nk, nv, hs)]
    if W < T:
        want.append(F.gdn_core(dev(qkvz[W:]), dev(ab[W:]), Hw, *args, Sw, dev(np.array([(cur + W) % NS], np.int32)), None, nk, nv, hs))
    got = F.gdn_prompt(dev(qkvz), dev(ab), Hp, *args, Sp, cur, nk, nv, hs)
    out = (cur + T) % NS
    # (the bound of the prompt against chained windows)
    assert rel_err(got.cpu().numpy(), torch.cat(want).cpu().numpy()) < 1e-4
    assert rel_err(Sp[out].cpu().numpy(), Sw[out].cpu().numpy()) < 1e-4
    for t in range(NS):
        if t != out:
            assert torch.equal(Sp[t].cpu(), torch.from_numpy(S0[t])), t
