"""Norm, rotary encoding and cache write of many tokens against 64 bits: both sides of the token counts where the kernel changes
(128, and two tokens a lane from 512 on), head counts that do not fill a warp or a block, tokens without a slot."""
import pytest
import torch
from types import SimpleNamespace as NS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("T,H,Hkv,D,norm", [(127, 4, 2, 128, True), (128, 4, 2, 128, True), (511, 3, 1, 64, True), (513, 9, 3, 64, True),
                                            (512, 64, 8, 128, True), (515, 5, 1, 256, False), (640, 33, 3, 128, True)])
def test_rows(T, H, Hkv, D, norm, dtype):
    from tinyserve_b200.kernels import ops
    g = torch.Generator().manual_seed(T + H)
    page, pages = 16, T // 16 + 2
    qkv = torch.randn(T, (H + 2 * Hkv) * D, generator=g).to(dtype).cuda()
    w = [(1 + 0.1 * torch.randn(D, generator=g)).to(dtype).cuda() if norm else None for _ in range(2)]
    pos = torch.randint(0, 4096, (T,), generator=g).int().cuda()
    slots = torch.randperm(pages * page, generator=g)[:T].int()
    slots[::7] = -1
    angles = torch.arange(4096).double()[:, None] * 10000.0 ** (-torch.arange(0, D, 2).double() / D)
    rot = NS(cos=angles.cos().float().cuda(), sin=angles.sin().float().cuda(), rotary_dim=D, interleaved=False)
    k, v = (torch.full((pages, Hkv, page, D), 7.0, dtype=dtype, device="cuda") for _ in range(2))
    q = ops.qk_norm_rope_kvwrite(qkv, pos, H, Hkv, D, rotary=rot, q_weight=w[0], k_weight=w[1], eps=1e-6, k_cache=k, v_cache=v,
                                 slot_mapping=slots.cuda(), page_size=page)
    x = qkv.double().view(T, H + 2 * Hkv, D)
    c, s = rot.cos.double()[pos.long()][:, None], rot.sin.double()[pos.long()][:, None]

    def turned(y, weight):
        if weight is not None:
            y = y * (y.square().mean(-1, keepdim=True) + 1e-6).rsqrt() * weight.double()
        a, b = y.chunk(2, -1)
        return torch.cat([a * c - b * s, b * c + a * s], -1)

    # one rounding of the result in bfloat16; a handful of operations in 32 bits
    unit = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -20
    wants = turned(x[:, :H], w[0]), turned(x[:, H:H + Hkv], w[1]), x[:, H + Hkv:]
    assert (q.view(T, H, D).double() - wants[0]).abs().max() <= unit * wants[0].abs().max()
    for cache, want in ((k, wants[1]), (v, wants[2])):
        full = torch.full((pages * page, Hkv, D), 7.0, dtype=torch.float64, device="cuda")
        kept = slots >= 0
        full[slots[kept].long().cuda()] = want[kept.cuda()]
        got = cache.transpose(1, 2).reshape(pages * page, Hkv, D).double()
        assert (got - full).abs().max() <= unit * want.abs().max()
