"""Attention whose slices meet in the shared memory of a cluster (qdecode.cu): every number of slices, slices without a position, the new row at the
edges of slices and turns, rotary tables off 16 bytes."""
import pytest
import torch

from ai_accel_studio_b200 import decode_step as ds

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("batch,hq,hkv,d,max_len,positions", [
    (1, 2, 1, 64, 192, (0, 15, 16, 23, 24, 127, 191)),       # eight slices of 16 or 32 positions, the last ones empty
    (1, 16, 2, 128, 191, (190,)),                            # just below: one slice
    (2, 32, 8, 128, 300, (5, 255, 299)),                     # six
    (3, 8, 8, 64, 1100, (1099,)),                            # five, several turns each
    (4, 16, 8, 128, 640, (127, 512)),                        # four
    (5, 8, 8, 64, 200, (3, 199)),                            # three
    (8, 8, 8, 128, 256, (129, 255)),                         # two
    (1, 3, 1, 64, 1025, (1023, 1024)),                       # a second turn in every slice
])
def test_slices_of_a_cluster(dtype, batch, hq, hkv, d, max_len, positions):
    g = torch.Generator(device="cuda").manual_seed(hq * d + max_len)
    rnd = lambda *shape: torch.empty(shape, device="cuda").normal_(0, 1, generator=g).to(dtype)
    ang = torch.rand(max_len, d, device="cuda", generator=g) * 6
    tables = torch.empty(2 * max_len * d + 1, dtype=dtype, device="cuda")
    for shift in (0, 1):                                     # the tables' first element on 16 bytes, and off
        cos, sin = (tables[shift + i * max_len * d:shift + (i + 1) * max_len * d].view(max_len, d).copy_(f(ang)) for i, f in enumerate((torch.cos, torch.sin)))
        for p in positions:
            q, k, v = rnd(batch, hq * d), rnd(batch, hkv * d), rnd(batch, hkv * d)
            kc, vc = rnd(batch, hkv, max_len, d), rnd(batch, hkv, max_len, d)
            kc[:, :, p:] = float("nan")
            vc[:, :, p:] = float("nan")
            kc2, vc2, q2 = kc.clone(), vc.clone(), q.clone()
            pos, status = torch.tensor([p], device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
            ws, scale = ds.attention_workspace(batch, hq, hkv, d, max_len, "cuda"), d ** -0.5
            got = ds.rope_attention(q, k, v, cos, sin, pos, kc, vc, scale, ws, status)
            ds.rope_append(q2, k, v, cos, sin, pos, kc2, vc2, d, status)
            assert torch.equal(kc[:, :, :p + 1], kc2[:, :, :p + 1]) and torch.equal(vc[:, :, :p + 1], vc2[:, :, :p + 1])
            assert torch.equal(got, ds.attention(q2, kc2, vc2, pos, scale, ws)) and int(status.item()) == 0
            n = p + 1
            kf, vf = (c[:, :, :n].double().repeat_interleave(hq // hkv, dim=1) for c in (kc, vc))
            qd = q2.double().reshape(batch, hq, d)
            score = torch.einsum("bhd,bhjd->bhj", qd, kf) * scale
            ref = torch.einsum("bhj,bhjd->bhd", torch.softmax(score, -1), vf)
            # fp32 dot products of d terms move an exponent by at most d 2^-24 sum |q k| scale, the exponential by a few 2^-22 of its argument; a relative
            # change of every weight by e changes the result by at most 2 e max |v|; then one rounding
            size = torch.einsum("bhd,bhjd->bhj", qd.abs(), kf.abs()).amax(-1) * scale
            e = d * 2.0 ** -24 * size + 2.0 ** -20 * (1 + score.abs().amax(-1)) + n * 2.0 ** -24
            tol = 2 * e[..., None] * vf.abs().amax(2).amax(-1)[..., None] + 2.0 ** (-11 if dtype == torch.float16 else -8) * ref.abs() * 1.01 + 2.0 ** -24
            assert bool(((got.double().reshape(batch, hq, d) - ref).abs() <= tol).all()), (p, shift)
