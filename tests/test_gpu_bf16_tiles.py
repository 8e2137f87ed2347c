"""The bf16 prefill product through each of its tile widths (256, 192, 128 and 64 weight rows): plain products, several matrices of one input,
GLU halves and column groups, at sizes that end inside a tile."""
import numpy as np
import pytest

import hybrid_oracle as orc
from hybrid_util import attn, config, rec, rel, weights, write_checkpoint

pytestmark = pytest.mark.gpu
SMS = 148


def width(M, rows, glu=False, groups=1):
    """the rule of kq_gemm_bf16: the cheapest number of waves; rows: of each matrix (padded to 64 where a GLU's output is)"""
    def cost(tn, weight):
        tiles = -(-rows[0] // (tn // 2)) if glu else sum(-(-n // tn) for n in rows)
        return -(-(-(-M // 128) * tiles * groups) // SMS) * weight
    return min(((256, 40), (192, 36), (128, 26), (64, 18)), key=lambda c: cost(*c))[0]


PLAIN = [(1000, 4600, 256), (2048, 4600, 256), (1000, 3000, 192), (300, 9000, 192), (900, 2200, 128), (300, 1100, 64)]


@pytest.mark.parametrize("M,N,tn", PLAIN)
@pytest.mark.parametrize("K", [64, 200])
def test_product(M, N, tn, K):
    """bf16 operands exactly, f32 sums of at most 200 terms (truncating: 2^-22 each)"""
    import torch

    from mesh_llm_b200 import ops

    assert width(M, [N]) == tn and torch.cuda.get_device_properties(0).multi_processor_count == SMS
    g = torch.Generator(device="cuda").manual_seed(M + N)
    w = torch.randn((N, K), generator=g, device="cuda").to(torch.bfloat16)
    x = torch.randn((M, K), generator=g, device="cuda").to(torch.bfloat16).float()
    got = ops.mul_mat_bf16(ops.upload_bf16(w), x, N, K).double()
    size = x.double().abs() @ w.double().abs().T
    assert ((got - x.double() @ w.double().T).abs() <= K * 2.0 ** -22 * size).all()


def test_layers_at_192_rows(tmp_path):
    """1000 tokens through layers whose every wide product takes tiles of 192 rows: two and three matrices of one input, gates by block (groups of 190
    rows), a GLU of 1700 (halves of 96, staging rows padded to 1728).  bf16 activations, as in the other tests of these layers"""
    import torch

    from mesh_llm_b200.engine import open_stage

    T = 1000
    cfg = config([rec(1710, 9, 4, ff=1700), attn(10, 128, 64, 128, 512, window=300)], width=64, vocab=96, scale=2.0)
    assert width(T, [1710, 1710]) == width(T, [190, 190], groups=9) == width(T, [1728], glu=True) == width(T, [1920, 576, 10]) == 192
    w = weights(cfg, 5)
    toks = np.random.default_rng(6).integers(0, cfg["vocab"], T).astype(np.int32)
    ref, res = orc.forward(cfg, w, toks)
    st = open_stage(write_checkpoint(tmp_path, cfg, w), "bfloat16", n_ctx=1024, n_seq=1, n_ubatch=T)
    buf = torch.zeros((len(res), T, cfg["width"]), device="cuda")
    st.trace_residual(buf)
    _, lg, _ = st.forward(tokens=torch.from_numpy(toks).cuda(), all_logits=True)
    st.trace_residual(None)
    st.synchronize()
    for i in range(len(res)):
        assert rel(buf[i].cpu().numpy(), res[i]).max() < 3e-2, (i, rel(buf[i].cpu().numpy(), res[i]).max())
    assert rel(lg.cpu().numpy(), ref).max() < 3e-2
    st.close()
