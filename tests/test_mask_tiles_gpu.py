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
