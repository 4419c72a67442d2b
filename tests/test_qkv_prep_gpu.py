"""Norm, rotation and cache store of a step's heads: many tokens (four heads per warp) against the same tokens in small steps (a
head per warp), vectors against rows that cannot be read in vectors, slots that are not stored, and the plain equations."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16


def _run(F, proj, ld, T, hq, hkv, D, rot, pos, slots, qn, kn, nb):
    q = torch.zeros(T, hq, D, dtype=BF16, device="cuda")
    kc, vc = torch.zeros(nb, hkv, 16, D, dtype=BF16, device="cuda"), torch.zeros(nb, hkv, D, 16, dtype=BF16, device="cuda")
    return q, kc, vc, lambda a, b: F.qkv_prep(_params(F, proj, ld, a, hq, hkv, D, rot, pos, slots, qn, kn, q, kc, vc, nb), b - a, D)


def _params(F, proj, ld, a, hq, hkv, D, rot, pos, slots, qn, kn, q, kc, vc, nb):
    p = F.QkvPrepParams()
    p.proj, p.q_norm, p.k_norm = proj.data_ptr() + 2 * a * ld, qn.data_ptr(), kn.data_ptr()
    p.positions, p.slot_mapping, p.q_out = pos[a:].data_ptr(), slots[a:].data_ptr(), q[a:].data_ptr()
    p.kcache, p.vcache, p.ld, p.hq, p.hkv, p.rotary_dim = kc.data_ptr(), vc.data_ptr(), ld, hq, hkv, rot
    p.eps, p.log2_theta, p.num_blocks = 1e-6, math.log2(1e6), nb
    return p


@pytest.mark.parametrize("pad", [0, 1, 6])
@pytest.mark.parametrize("D,hq,hkv,rot", [(256, 24, 4, 64), (256, 3, 1, 256), (128, 16, 4, 32), (64, 6, 1, 16), (64, 5, 2, 64)])
def test_forms_agree(D, hq, hkv, rot, pad):
    from tileinfer_b200.models.reference_cpu import rmsnorm, rope_partial
    from tileinfer_b200.ops import functional as F
    F.L()
    g = torch.Generator(device="cuda").manual_seed(D + hq + pad)
    T, nb, ld = 301, 40, hq * 2 * D + 2 * hkv * D + pad
    proj = torch.randn(T, ld, generator=g, device="cuda").to(BF16)
    pos = torch.randint(0, 30000, (T,), generator=g, device="cuda", dtype=torch.int32)
    slots = torch.randperm(nb * 16, generator=g, device="cuda")[:T].clone()
    slots[7::50] = -1
    qn, kn = ((torch.randn(D, generator=g, device="cuda") * 0.1).to(BF16) for _ in range(2))
    args = (hq, hkv, D, rot, pos, slots, qn, kn, nb)
    q, kc, vc, run = _run(F, proj, ld, T, *args)
    run(0, T)
    q2, kc2, vc2, run = _run(F, proj, ld, T, *args)
    for a in range(0, T, 100):
        run(a, min(T, a + 100))
    torch.cuda.synchronize()
    assert torch.equal(q, q2) and torch.equal(kc, kc2) and torch.equal(vc, vc2)
    rows = proj[:, :ld - pad].float()
    qk = rows[:, :hq * 2 * D].view(T, hq, 2, D)[:, :, 0]
    k, v = rows[:, hq * 2 * D:].view(T, 2, hkv, D).unbind(1)
    turn = lambda x, w: rope_partial(rmsnorm(x, w, 1e-6).to(BF16).float(), pos, rot, 1e6)  # noqa: E731
    # angles up to 30000 radians in fp32: 2^-9 off; results rounded to bf16: 2^-9 relative of values up to about 5
    assert float((q.float() - turn(qk, qn)).abs().max()) < 5 * 2.0 ** -8
    ok = slots >= 0
    at = slots[ok]
    assert float((kc.transpose(1, 2).reshape(nb * 16, hkv, D)[at].float() - turn(k, kn)[ok]).abs().max()) < 5 * 2.0 ** -8
    assert torch.equal(vc.permute(0, 3, 1, 2).reshape(nb * 16, hkv, D)[at].float(), v[ok])
    free = torch.ones(nb * 16, dtype=torch.bool, device="cuda")
    free[at] = False
    assert not bool(kc.transpose(1, 2).reshape(nb * 16, hkv, D)[free].any())
