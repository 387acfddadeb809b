"""Tile lists of a key mask: the joint call's (extra blocks of the prologue launch) and the attention-only call's (a
kernel of its own) against float64 attention over the open keys."""
import numpy as np
import pytest

from zdraw_b200 import _lib, mattn

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


# Tiles of 128 keys, classified 256 at a time: one key, the ragged end of the first tile, one whole tile, the last tile
# of a chunk, the first of the next, a partly open last tile; an image of its own mask and one shared by two.
@pytest.mark.parametrize("tokens,open_keys,batch,shared", [
    (1, [(0, 1)], 1, True), (130, [(127, 130)], 2, True), (256, [(128, 256)], 1, True),
    (1153, [(5, 6), (512, 640), (1152, 1153)], 2, False), (32901, [(3, 7), (32639, 32770), (32896, 32901)], 1, True)])
def test_lists_of_both_launches(tokens, open_keys, batch, shared):
    ctx = mattn.Context(0)
    g = torch.Generator(device="cuda").manual_seed(tokens)
    shape = (batch, tokens, 1, 128)
    q, k, v = (torch.randn(shape, generator=g, device="cuda").half() for _ in range(3))
    ones = torch.ones(128, device="cuda")
    cos, sin = torch.ones((tokens, 128), device="cuda"), torch.zeros((tokens, 128), device="cuda")
    stride = 0 if shared else (tokens + 3) // 4 * 4
    mask = torch.full((1 if shared else batch, stride or tokens), float("-inf"), device="cuda")
    for i in range(mask.shape[0]):
        for a, b in open_keys[i:]:  # the second image's own mask leaves the first range closed
            mask[i, a:b] = 0.0
    p = _lib.AttnParams(batch=batch, tokens=tokens, heads=1, head_dim=128, txt_tokens=0, in_dtype=1, out_dtype=1,
                        qk_layout=1, has_key_mask=1, norm_eps=1e-6, mask_batch_stride=stride)
    got = torch.full(shape, float("nan"), device="cuda", dtype=torch.float16)
    ctx.joint_attention(q, k, v, ones, ones, ones, ones, cos, sin, got, p, key_mask=mask)
    q16, k16 = (torch.empty((batch, 1, tokens, 128), device="cuda", dtype=torch.float16) for _ in range(2))
    ctx.qk_norm_rope(q, k, ones, ones, ones, ones, cos, sin, q16, k16, p)
    alone = torch.full_like(got, float("nan"))
    ctx.run_on_handles(q16, k16, v, alone, p, key_mask=mask)
    torch.cuda.synchronize()
    assert ctx.last_status() == 0
    assert torch.equal(got, alone)
    for i in range(batch):
        keys = torch.nonzero(mask[0 if shared else i, :tokens] == 0.0)[:, 0]
        s = q16[i, 0].double() @ k16[i, 0][keys].double().T / np.sqrt(128.0)
        want = torch.softmax(s, -1) @ v[i, :, 0][keys].double()
        # P and O are rounded to half (2^-11 each) and |v| <= about 4: the bound of the attention tests, 1e-2
        assert (got[i, :, 0].double() - want).abs().max() <= 1e-2
    ctx.deinit()


# The three kinds of blocks of one prologue launch at once: a mask of each image, q and k, an f32 V of a wider row.
@pytest.mark.parametrize("tokens,heads,batch,extra", [(1, 1, 1, 8), (129, 3, 2, 64), (700, 2, 3, 24), (257, 9, 2, 0)])
def test_mask_and_cast_ride_in_one_prologue_launch(tokens, heads, batch, extra):
    ctx = mattn.Context(0)
    g = torch.Generator(device="cuda").manual_seed(tokens)
    ld = heads * 128 + extra
    full = torch.randn((3, batch, tokens, ld), generator=g, device="cuda")
    full[..., heads * 128:] = float("nan")  # the columns between the rows belong to others
    q, k, v = full
    w = [torch.rand(128, generator=g, device="cuda") * 0.4 + 0.8 for _ in range(4)]
    angle = torch.rand((tokens, 64), generator=g, device="cuda").repeat_interleave(2, 1) * 6.0
    cos, sin = angle.cos(), angle.sin()
    stride = (tokens + 3) // 4 * 4
    mask = torch.where(torch.rand((batch, stride), generator=g, device="cuda") < 0.3, float("-inf"), 0.0)
    mask[:, tokens - 1] = 0.0
    mask[0, :128 * ((tokens - 1) // 128)] = float("-inf")  # whole tiles of the first image
    p = _lib.AttnParams(batch=batch, tokens=tokens, heads=heads, head_dim=128, txt_tokens=tokens // 3, in_dtype=3, out_dtype=3,
                        qk_layout=1, has_key_mask=1, norm_eps=1e-6, mask_batch_stride=stride, ld_q=ld, ld_k=ld, ld_v=ld)
    got, alone = (torch.full((batch, tokens, heads, 128), float("nan"), device="cuda") for _ in range(2))
    ctx.joint_attention(q, k, v, *w, cos, sin, got, p, key_mask=mask)
    q16, k16 = (torch.empty((batch, heads, tokens, 128), device="cuda", dtype=torch.float16) for _ in range(2))
    ctx.qk_norm_rope(q, k, *w, cos, sin, q16, k16, p)
    ctx.run_on_handles(q16, k16, v, alone, p, key_mask=mask)  # the cast and the lists in launches of their own
    torch.cuda.synchronize()
    assert ctx.last_status() == 0
    assert torch.equal(got, alone)
    vh = v[..., :heads * 128].reshape(batch, tokens, heads, 128).permute(0, 2, 1, 3).double()
    s = q16.double() @ k16.double().transpose(-1, -2) / np.sqrt(128.0) + mask[:, None, None, :tokens].double()
    want = (torch.softmax(s, -1) @ vh).permute(0, 2, 1, 3)
    # P and V are rounded to half (2^-11 each) and |v| <= about 5: the bound of the attention tests, 1e-2
    assert (got - want).abs().max() <= 1e-2
    ctx.deinit()
