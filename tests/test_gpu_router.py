"""The router of a micro-batch in its forms, sum for sum the same: blocks of 32 tokens x 32 experts where those are fewer waves than tiles, tiles of 8 x 8 per warp from 256 tiles
on, a warp per pair below; and norm, logits and choice in one launch for few rows."""
import numpy as np
import pytest

from oracle import binding as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("E,T", [(20, 1030), (8, 2049), (130, 129)])
def test_both_forms_route_alike(E, T):
    """one layer of experts over T tokens at once (tiles, the last ones of them part empty) and in four parts (warps per pair).  The logits of the two
    forms are equal sum for sum, so a token takes the same experts.  What differs are sums of the products in another order, which put Q8 codes beside a
    tie on its other side: one code in a hundred moved by 1 / 127 of a block's largest value, which is about three times its rms, is 2.4e-3 of a row, in
    each of the layer's four quantisers.  A wrong expert moves a row by its whole expert part"""
    import torch

    from mesh_llm_b200.stage import Stage

    cfg = dict(n_layer=1, n_embd=512, n_head=8, n_head_kv=2, head_dim=64, n_ff=0, n_vocab=256, n_ctx=2304, n_expert=E, n_expert_used=4, n_ff_exp=256, qk_norm=1)
    part = dict(layer_begin=0, layer_end=1, has_embd=0, has_output=0)
    m = orc.Model(**cfg)
    m.generate(3)
    st = Stage(**cfg, **part, n_ubatch=T)
    for n in orc.Model(**cfg, **part).tensor_names():
        st.set_tensor(n, *m.tensor(n)[:2])
    x = torch.from_numpy(np.random.default_rng(E).standard_normal((T, cfg["n_embd"])).astype(np.float32)).cuda()
    whole = st.forward(hidden_in=x, n_seq=1, T=T, pos0=0)[0].double().clone()
    step = -(-T // 4)
    parts = torch.cat([st.forward(hidden_in=x[i:i + step].contiguous(), n_seq=1, T=min(step, T - i), pos0=i)[0].double().clone() for i in range(0, T, step)])
    st.close()
    change = whole - x.double()  # what the layer adds
    assert float((whole - parts).norm(dim=1).max() / change.norm(dim=1).mean()) <= 2e-2


@pytest.mark.parametrize("E,T,h", [(256, 256, 256), (250, 260, 768), (33, 1025, 512), (250, 520, 768), (62, 1801, 512), (256, 1025, 256)])
def test_blocks_of_many_tokens(E, T, h):
    """tiles (the first three) and the router's block form (one wave of blocks, full and with its last ones part empty, and two waves): the same
    experts as a warp per pair or the one launch take, and the same bound"""
    import torch

    from mesh_llm_b200.stage import Stage

    cfg = dict(n_layer=1, n_embd=h, n_head=4, n_head_kv=2, head_dim=64, n_ff=0, n_vocab=256, n_ctx=2048, n_expert=E, n_expert_used=2, n_ff_exp=256, qk_norm=1)
    part = dict(layer_begin=0, layer_end=1, has_embd=0, has_output=0)
    m = orc.Model(**cfg)
    m.generate(5)
    st = Stage(**cfg, **part, n_ubatch=T)
    for n in orc.Model(**cfg, **part).tensor_names():
        st.set_tensor(n, *m.tensor(n)[:2])
    x = torch.from_numpy(np.random.default_rng(T).standard_normal((T, h)).astype(np.float32)).cuda()
    whole = st.forward(hidden_in=x, n_seq=1, T=T, pos0=0)[0].double().clone()
    step = 31  # at most 128 tiles: the other forms
    parts = torch.cat([st.forward(hidden_in=x[i:i + step].contiguous(), n_seq=1, T=min(step, T - i), pos0=i)[0].double().clone() for i in range(0, T, step)])
    st.close()
    change = whole - x.double()
    assert float((whole - parts).norm(dim=1).max() / change.norm(dim=1).mean()) <= 2e-2


@pytest.mark.parametrize("E,h,few,many", [(128, 1024, 24, 25), (200, 1024, 16, 17), (16, 512, 8, 9)])
def test_one_launch_routing_of_a_few_rows(E, h, few, many):
    """on both sides of the number of rows up to which norm, logits and choice are one launch (three behind it): the same experts as six rows at a time take, and the same bound"""
    import torch

    from mesh_llm_b200.stage import Stage

    cfg = dict(n_layer=1, n_embd=h, n_head=4, n_head_kv=2, head_dim=64, n_ff=0, n_vocab=256, n_ctx=64, n_expert=E, n_expert_used=4, n_ff_exp=256, qk_norm=1)
    part = dict(layer_begin=0, layer_end=1, has_embd=0, has_output=0)
    m = orc.Model(**cfg)
    m.generate(7)
    st = Stage(**cfg, **part, n_ubatch=32)
    for n in orc.Model(**cfg, **part).tensor_names():
        st.set_tensor(n, *m.tensor(n)[:2])
    x = torch.from_numpy(np.random.default_rng(E).standard_normal((many, h)).astype(np.float32)).cuda()
    launches = {}
    for T in (few, many):
        before = st.kernel_launches()
        rows = x[:T].contiguous()
        whole = st.forward(hidden_in=rows, n_seq=1, T=T, pos0=0)[0].double().clone()
        launches[T] = st.kernel_launches() - before
        parts = torch.cat([st.forward(hidden_in=rows[i:i + 6].contiguous(), n_seq=1, T=min(6, T - i), pos0=i)[0].double().clone() for i in range(0, T, 6)])
        change = whole - rows.double()
        assert float((whole - parts).norm(dim=1).max() / change.norm(dim=1).mean()) <= 2e-2
    st.close()
    if few > 8:
        assert launches[many] == launches[few] + 2
