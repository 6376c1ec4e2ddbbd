"""The grouped GEMMs' edges that come from the weights being converted into tensor memory: an odd number of channel tiles (the last item of
down has one), blocks of few and of many picks in turn on one SM (they take one or both accumulator slots), a caller's row blocks of
more than one tile, and scales that the fused conversion cannot take. Against the CPU checker; fp16 operands, gate as in test_prefill_gpu."""
import numpy as np
import pytest

from helpers import HostLayer, errors
from hecate_b200 import synth

pytestmark = pytest.mark.gpu
NORM_REL = 2e-3


def _run(oracle, hl, R, sel, rw, scale=1.0):
    import torch
    from hecate_b200 import moe
    dev = torch.device("cuda:0")
    tabs = hl.upload(dev)
    x = (synth.activations(1, 0, R, hl.H) * scale).astype(np.float16)
    ex, sh = hl.oracle_experts(oracle)
    ref = oracle.moe_forward(hl.H, hl.I, hl.group, x, sel, rw, 0, ex, sh, mode=1)
    n = len(ex)
    ws = moe.prefill_workspace(R, 8, n, hl.H, hl.I, dev)
    out = torch.zeros(R, hl.H, device=dev)
    moe.prefill(tabs, torch.from_numpy(x).to(dev), torch.from_numpy(sel).to(dev), torch.from_numpy(rw).to(dev), out, ws, n_local=n)
    assert moe.ws_status(ws) == 0
    return errors(out.cpu().numpy(), ref)


@pytest.mark.parametrize("group", [0, 128])
@pytest.mark.parametrize("H,I", [(384, 512), (640, 384)])
def test_odd_channel_tiles_and_blocks_of_all_sizes_on_one_sm(oracle, H, I, group):
    """Zipf routing over 64 experts: several hundred items of 1 .. 128 picks, more than one per SM."""
    hl = HostLayer(3, 0, H, I, range(64), group, True)
    R = 700
    sel, rw = synth.zipf_routing(5, 0, R, 64, 8, 1.3)
    e = _run(oracle, hl, R, sel, rw)
    assert e[2] < NORM_REL, e


def test_scales_beyond_the_fused_conversion(oracle):
    """bf16 scales of 2048 and more (as far as the fp16 weights reach) in some column groups of some experts' down matrices."""
    hl = HostLayer(4, 0, 256, 256, range(8), 128, False)
    for k, d in enumerate(hl.ex):
        if k % 2:
            d["ds"] = d["ds"].copy()
            d["ds"][k % d["ds"].shape[0]] = (2048.0, 2720.0, 4000.0, 8000.0)[k // 2]
    sel, rw = synth.zipf_routing(6, 0, 200, 8, 8, 0.0)
    e = _run(oracle, hl, 200, sel, rw)
    assert np.isfinite(e[2]) and e[2] < NORM_REL, e


@pytest.mark.parametrize("offset", [0, 1, 2, 3])
@pytest.mark.parametrize("picks", [128, 129, 200, 256])
def test_row_blocks_of_a_caller_up_to_256_picks(oracle, picks, offset):
    """The table may start on any 4-byte boundary (a part of a larger int32 buffer)."""
    import torch
    from hecate_b200 import moe
    dev = torch.device("cuda:0")
    H, I = 256, 128
    hl = HostLayer(7, 0, H, I, range(2), 0, False)
    tabs = hl.upload(dev)
    x = synth.activations(1, 0, picks, H).astype(np.float16)
    # every row picks expert 0, the first five also expert 1
    sel = np.full((picks, 8), 100, dtype=np.int64)
    sel[:, 0] = 0
    sel[:5, 1] = 1
    rw = np.full((picks, 8), 0.125, dtype=np.float16)
    ex, _ = hl.oracle_experts(oracle)
    ref = oracle.moe_forward(H, I, 0, x, sel, rw, 0, ex, None, mode=1)
    tok = torch.cat([torch.arange(picks), torch.arange(5)]).to(torch.int32).to(dev)
    eid = torch.cat([torch.zeros(picks), torch.ones(5)]).to(torch.int32).to(dev)
    wt = torch.full((picks + 5,), 0.125, dtype=torch.float32, device=dev)
    buf = torch.zeros(8 + offset, dtype=torch.int32, device=dev)
    rbt = buf[offset:].view(2, 4)
    rbt.copy_(torch.tensor([[0, 0, picks, 0], [1, picks, 5, 0]]))
    assert rbt.data_ptr() % 16 == 4 * offset
    out = torch.zeros(picks, H, device=dev)
    t = tabs.tabs
    moe.moe4t_forward(torch.from_numpy(x).to(dev), tok, eid, wt, rbt, t["gate_w"], t["up_w"], t["down_w"], t["gate_s"], t["up_s"], t["down_s"],
                      *moe.moe4t_scratch(dev, picks + 5, H, I), out, I=I)
    e = errors(out.cpu().numpy(), ref)
    assert e[2] < NORM_REL, e
