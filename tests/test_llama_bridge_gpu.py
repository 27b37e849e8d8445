"""The llama.cpp bridge's entry points (include/polarquant_llama_abi.h) against the numpy
restatement of the bridge's kernels, through the C ABI."""

import numpy as np
import pytest
import torch

from oracle import llama_bridge_oracle as LO

pytestmark = pytest.mark.gpu

# Indices may differ from the float64 restatement only where the direction sits this close to
# the midpoint of the two candidate centroids (float32 rotation and division on the device).
INDEX_WINDOW = 1e-6
# north_star tolerance for attention outputs.
ATTN_ATOL = 2e-3


def codebook_for(n_levels, rng):
    cb = np.sort(rng.normal(0.0, 0.09, n_levels)).astype(np.float32)
    return cb


def orthogonal(d, rng):
    q, _ = np.linalg.qr(rng.standard_normal((d, d)))
    return q.astype(np.float32)


def explained(direction, cb, got, want):
    """Mismatching indices whose two candidates are equally near within the window."""
    bad = np.argwhere(got != want)
    unexplained = 0
    worst = 0.0
    for n, j in bad:
        gap = abs(abs(direction[n, j] - cb[got[n, j]]) - abs(direction[n, j] - cb[want[n, j]]))
        worst = max(worst, gap)
        if gap > 2 * INDEX_WINDOW:
            unexplained += 1
    return len(bad), unexplained, worst


# n >= 4096 at head dim 64 / 128 takes the kernel with R transposed in shared memory, or, above a wave of its CTAs, the
# tensor-core kernel; everything else the kernel with one vector (from 768 on four) per CTA
@pytest.mark.parametrize("d,n_levels,n", [(128, 16, 767), (256, 16, 768), (64, 4, 769), (128, 16, 1000), (128, 4, 37), (64, 16, 513), (64, 8, 3),
                                          (96, 16, 200), (256, 16, 65), (130, 8, 9), (128, 16, 1),
                                          (128, 16, 20_003), (64, 4, 4096), (64, 16, 70_001), (128, 8, 4097)])
def test_compress_vs_oracle(d, n_levels, n):
    from polarquant_kv import llama_bridge as LB
    rng = np.random.default_rng(d * 131 + n_levels * 7 + n)
    x = (rng.standard_normal((n, d)) * rng.uniform(0.05, 30.0, (n, 1))).astype(np.float32)
    if n > 2:
        x[1] = 0.0                                         # radius 0: every direction is 0
    R, cb = orthogonal(d, rng), codebook_for(n_levels, rng)
    radius, packed = LB.compress(torch.from_numpy(x).cuda(), torch.from_numpy(R).cuda(), torch.from_numpy(cb).cuda())
    radius, packed = radius.cpu().numpy(), packed.cpu().numpy()
    want_radius, want_packed, direction = LO.compress(x, R, cb)
    np.testing.assert_allclose(radius, want_radius, rtol=2e-6, atol=1e-30)
    got_idx, want_idx = LO.unpack(packed, 16), LO.unpack(want_packed, 16)
    n_bad, n_unexplained, worst = explained(direction, cb.astype(np.float64), got_idx, want_idx)
    print(f"compress d={d} levels={n_levels} n={n}: {n_bad} of {got_idx.size} indices differ, "
          f"{n_unexplained} unexplained, widest gap {worst:.2e}")
    assert n_unexplained == 0
    assert n_bad <= max(2, got_idx.size // 2000)
    if n > 2:
        zero_level = int(np.argmin(np.abs(cb)))
        assert (got_idx[1] == zero_level).all() and radius[1] == 0.0


@pytest.mark.parametrize("d,rows", [(128, 32), (64, 7), (96, 3), (256, 40), (1024, 2)])
def test_rotate_and_inverse_vs_oracle(d, rows):
    from polarquant_kv import llama_bridge as LB
    rng = np.random.default_rng(d + rows)
    x = rng.standard_normal((rows, d)).astype(np.float32)
    R = orthogonal(d, rng)
    xr = LB.rotate_query(torch.from_numpy(x).cuda(), torch.from_numpy(R).cuda())
    np.testing.assert_allclose(xr.cpu().numpy(), LO.rotate(x, R), atol=2e-5)
    back = LB.inverse_rotate(xr, torch.from_numpy(R).cuda())
    np.testing.assert_allclose(back.cpu().numpy(), LO.inverse_rotate(xr.cpu().numpy(), R), atol=2e-5)
    np.testing.assert_allclose(back.cpu().numpy(), x, atol=1e-4)


def random_cache(hkv, s, d, n_levels, rng):
    idx = rng.integers(0, n_levels, (hkv, s, d), dtype=np.uint8)
    packed = (idx[..., 0::2] | (idx[..., 1::2] << 4)).astype(np.uint8)
    radius = rng.uniform(0.2, 12.0, (hkv, s)).astype(np.float32)
    return packed, radius


@pytest.mark.parametrize("hq,hkv,s,d,n_levels", [
    (8, 2, 1, 128, 16), (8, 2, 33, 128, 16), (32, 8, 1000, 128, 16), (32, 8, 20000, 128, 16),
    (4, 4, 4097, 64, 16), (16, 2, 777, 64, 4), (6, 2, 300, 96, 8), (12, 2, 2500, 128, 16),
    (8, 1, 5000, 256, 16), (2, 1, 260, 130, 16), (2, 2, 90, 512, 16), (1, 1, 70, 1024, 4),
    (16, 2, 131072, 128, 16)])
def test_fused_attention_vs_oracle(hq, hkv, s, d, n_levels):
    from polarquant_kv import llama_bridge as LB
    rng = np.random.default_rng(hq * 1009 + s * 13 + d + n_levels)
    cb = codebook_for(n_levels, rng)
    pk, kr = random_cache(hkv, s, d, n_levels, rng)
    pv, vr = random_cache(hkv, s, d, n_levels, rng)
    q = (rng.standard_normal((hq, d)) * 1.5).astype(np.float32)
    scale = 1.0 / np.sqrt(d)
    dev = lambda a: torch.from_numpy(a).cuda()
    out = LB.fused_attention(dev(q), dev(pk), dev(kr), dev(pv), dev(vr), dev(cb), scale).cpu().numpy()
    want = LO.fused_attention(q, pk, kr, pv, vr, cb, n_levels, scale)
    err = np.abs(out - want).max()
    print(f"attention hq={hq} hkv={hkv} s={s} d={d} levels={n_levels}: max abs err {err:.2e} "
          f"(output scale {np.abs(want).max():.3f})")
    assert err <= ATTN_ATOL
    assert err <= 1e-4 * max(1.0, np.abs(want).max())


def test_peaked_scores_and_large_radii():
    """One token dominates by far; the running maximum moves upward across tiles and slices."""
    from polarquant_kv import llama_bridge as LB
    rng = np.random.default_rng(5)
    hq, hkv, s, d, n_levels = 8, 2, 9000, 128, 16
    cb = codebook_for(n_levels, rng)
    pk, kr = random_cache(hkv, s, d, n_levels, rng)
    pv, vr = random_cache(hkv, s, d, n_levels, rng)
    kr = (kr * np.linspace(0.1, 40.0, s, dtype=np.float32)[None, :]).astype(np.float32)
    q = (rng.standard_normal((hq, d)) * 4.0).astype(np.float32)
    dev = lambda a: torch.from_numpy(a).cuda()
    out = LB.fused_attention(dev(q), dev(pk), dev(kr), dev(pv), dev(vr), dev(cb), 1.0 / np.sqrt(d)).cpu().numpy()
    want = LO.fused_attention(q, pk, kr, pv, vr, cb, n_levels, 1.0 / np.sqrt(d))
    assert np.isfinite(out).all()
    assert np.abs(out - want).max() <= ATTN_ATOL


def test_state_and_whole_sequence_of_calls():
    """polarquant_init_c's state, then compress K and V, rotate q, attend, rotate back — the order
    the bridge calls them in — against float64 arithmetic on the same codes."""
    from polarquant_kv import llama_bridge as LB
    rng = np.random.default_rng(11)
    d, hkv, hq, s = 128, 4, 16, 700
    with LB.State(d, hkv, hq, n_layers=2, n_kv_max=1024, n_bits=4) as st:
        f = st.fields
        assert (f.enabled, f.n_bits, f.n_levels, f.head_dim, f.n_kv_heads, f.n_q_heads, f.n_layers, f.n_kv_max) == \
            (True, 4, 16, d, hkv, hq, 2, 1024)
        cb = st.device_tensor(f.codebook, 16)
        R = st.device_tensor(f.rotation, d * d).view(d, d)
        Rn = R.cpu().numpy().astype(np.float64)
        np.testing.assert_allclose(Rn @ Rn.T, np.eye(d), atol=2e-5)
        cbn = cb.cpu().numpy()
        assert cbn[0] == np.float32(-0.1547) and cbn[15] == np.float32(0.1947) and (np.diff(cbn) > 0).all()

        k = (rng.standard_normal((hkv * s, d)) * 2.0).astype(np.float32)
        v = rng.standard_normal((hkv * s, d)).astype(np.float32)
        q = rng.standard_normal((hq, d)).astype(np.float32)
        k_radius, k_packed = LB.compress(torch.from_numpy(k).cuda(), R, cb)
        v_radius, v_packed = LB.compress(torch.from_numpy(v).cuda(), R, cb)
        q_rot = LB.rotate_query(torch.from_numpy(q).cuda(), R)
        scale = 1.0 / np.sqrt(d)
        out_rot = LB.fused_attention(q_rot, k_packed.view(hkv, s, d // 2), k_radius.view(hkv, s),
                                     v_packed.view(hkv, s, d // 2), v_radius.view(hkv, s), cb, scale)
        out = LB.inverse_rotate(out_rot, R).cpu().numpy()

        want_rot = LO.fused_attention(LO.rotate(q, Rn), k_packed.view(hkv, s, d // 2).cpu().numpy(),
                                      k_radius.view(hkv, s).cpu().numpy(), v_packed.view(hkv, s, d // 2).cpu().numpy(),
                                      v_radius.view(hkv, s).cpu().numpy(), cbn, 16, scale)
        want = LO.inverse_rotate(want_rot, Rn)
        assert np.abs(out - want).max() <= ATTN_ATOL
        # and the codec does its job: close to exact attention over the uncompressed K and V
        kk, vv = k.reshape(hkv, s, d).astype(np.float64), v.reshape(hkv, s, d).astype(np.float64)
        exact = np.empty((hq, d))
        for h in range(hq):
            sc = kk[h // (hq // hkv)] @ q[h].astype(np.float64) * scale
            w = np.exp(sc - sc.max())
            exact[h] = (w / w.sum()) @ vv[h // (hq // hkv)]
        cos = (out * exact).sum() / (np.linalg.norm(out) * np.linalg.norm(exact))
        assert cos > 0.9
    for bits, levels in ((3, 8), (2, 4), (7, 16)):
        with LB.State(64, 2, 4, 1, 16, bits) as st:
            assert st.fields.n_levels == levels


def test_arguments_the_bridge_cannot_serve_are_reported():
    from polarquant_kv import llama_bridge as LB
    x = torch.zeros(4, 127, device="cuda")
    with pytest.raises(ValueError, match="even"):
        LB.compress(x, torch.zeros(127, 127, device="cuda"), torch.zeros(16, device="cuda"))
    q = torch.zeros(6, 64, device="cuda")
    pk = torch.zeros(4, 10, 32, dtype=torch.uint8, device="cuda")
    r = torch.ones(4, 10, device="cuda")
    with pytest.raises(ValueError, match="multiple"):
        LB.fused_attention(q, pk, r, pk, r, torch.zeros(16, device="cuda"), 1.0)
    with pytest.raises(ValueError, match="n_levels"):
        LB.fused_attention(torch.zeros(4, 64, device="cuda"), pk, r, pk, r, torch.zeros(17, device="cuda"), 1.0)


# edges of the tensor-core compress kernel: its smallest size, several tiles per CTA with a ragged last one, and
# codebooks its bucket table cannot hold (descending, levels in one bucket), which are scanned
@pytest.mark.parametrize("d,n,book", [(128, 4095, "normal"), (64, 513, "normal"), (128, 4096, "normal"), (64, 4097, "normal"), (128, 60_011, "normal"),
                                      (64, 130_049, "normal"), (128, 4500, "descending"), (64, 4500, "narrow")])
def test_compress_tensor_core_edges_vs_oracle(d, n, book):
    from polarquant_kv import _ext
    from polarquant_kv import llama_bridge as LB
    rng = np.random.default_rng(n + d)
    x = (rng.standard_normal((n, d)) * np.exp(rng.uniform(-30, 30, (n, 1)))).astype(np.float32)
    x[1] = 0.0
    R, cb = orthogonal(d, rng), codebook_for(16, rng)
    if book == "descending":
        cb = cb[::-1].copy()
    elif book == "narrow":
        cb = np.sort((0.02 * rng.standard_normal(16)).astype(np.float32))
    radius, packed = LB.compress(torch.from_numpy(x).cuda(), torch.from_numpy(R).cuda(), torch.from_numpy(cb).cuda())
    want_radius, want_packed, direction = LO.compress(x, R, cb)
    # six bfloat16 product terms (2^-24 each dropped) and a few truncating float32 accumulations: a few units of 2^-23
    np.testing.assert_allclose(radius.cpu().numpy(), want_radius, rtol=2e-6, atol=1e-30)
    got, want = LO.unpack(packed.cpu().numpy(), 16), LO.unpack(want_packed, 16)
    n_bad, n_unexplained, worst = explained(direction, cb.astype(np.float64), got, want)
    assert n_unexplained == 0 and n_bad <= max(2, got.size // 2000), (n_bad, n_unexplained, worst)
    assert _ext.poll_device_errors() == 0


# edges of the kernel for head dims 64 and 128: every group width (missing heads masked), tiles of one token, slices
@pytest.mark.parametrize("hq,hkv,s", [(1, 1, 31), (2, 2, 32), (6, 3, 129), (3, 1, 64), (7, 1, 1000), (10, 2, 513),
                                      (20, 1, 300), (5, 5, 4099), (2, 1, 70_001),
                                      (14, 2, 512), (14, 2, 513), (9, 1, 200), (40, 8, 1), (700, 700, 32), (700, 350, 64), (700, 350, 65), (700, 700, 65)])
@pytest.mark.parametrize("d", [64, 128])
def test_fused_attention_group_widths_vs_oracle(hq, hkv, s, d):
    from polarquant_kv import _ext
    from polarquant_kv import llama_bridge as LB
    rng = np.random.default_rng(hq * 7 + hkv + s + d)
    cb = codebook_for(16, rng)
    pk, kr = random_cache(hkv, s, d, 16, rng)
    pv, vr = random_cache(hkv, s, d, 16, rng)
    q = (rng.standard_normal((hq, d)) * 1.5).astype(np.float32)
    dev = lambda a: torch.from_numpy(a).cuda()
    out = LB.fused_attention(dev(q), dev(pk), dev(kr), dev(pv), dev(vr), dev(cb), 0.1).cpu().numpy()
    want = LO.fused_attention(q, pk, kr, pv, vr, cb, 16, 0.1)
    # float32 throughout: scores of a few tens carry about 1e-5, which the weights inherit
    assert np.abs(out - want).max() <= 1e-4 * max(1.0, np.abs(want).max())
    assert _ext.poll_device_errors() == 0


def fp32_chain(x, R, cb):
    """The bridge's compress in float32 as a chain: k ascending per coordinate, one rounding per multiply-add; squares as a
    tree (element t with t + D/2, then + D/4, ...); quotient; the first of the closest levels.  (A float64 sum rounded to
    float32 is the fused operation's result but for ties of the double rounding, one in 2^29.)"""
    n, d = x.shape
    xd, Rd = torch.from_numpy(x).cuda().double(), torch.from_numpy(R).cuda().double()
    acc = torch.zeros(n, d, device="cuda")
    for k in range(d):
        acc = (acc.double() + xd[:, k:k + 1] * Rd[:, k][None]).float()
    v = acc.cpu().numpy()
    with np.errstate(all="ignore"):
        t = v * v
        while t.shape[1] > 1:
            t = t[:, :t.shape[1] // 2] + t[:, t.shape[1] // 2:]
        radius = np.sqrt(t[:, 0])
        direction = np.where(radius[:, None] > np.float32(1e-30), v / radius[:, None], np.float32(0))
        best, dist = np.zeros((n, d), np.uint8), np.full((n, d), 1e30, np.float32)
        for level in range(len(cb)):
            far = np.abs(direction - cb[level])
            closer = far < dist
            best[closer], dist[closer] = level, far[closer]
    return radius, (best[:, 0::2] | (best[:, 1::2] << 4)).astype(np.uint8)


def kv_like(n, d, rng):
    scale = np.exp(rng.standard_normal(d))
    scale[rng.choice(d, 2, replace=False)] *= 10.0
    return (rng.standard_normal((n, d)) * scale).astype(np.float32)


@pytest.mark.parametrize("d,n", [(128, 20_003), (64, 30_001), (128, 4096)])
@pytest.mark.parametrize("kind", ["kv", "normal", "positive"])
def test_radius_is_as_close_to_64_bits_as_an_fp32_chain(d, n, kind):
    from polarquant_kv import llama_bridge as LB
    rng = np.random.default_rng(n + d)
    x = kv_like(n, d, rng) if kind == "kv" else rng.standard_normal((n, d)).astype(np.float32)
    if kind == "positive":
        x = np.abs(x) + np.float32(1)
    R, cb = orthogonal(d, rng), codebook_for(16, rng)
    radius, _ = LB.compress(torch.from_numpy(x).cuda(), torch.from_numpy(R).cuda(), torch.from_numpy(cb).cuda())
    chain, _ = fp32_chain(x, R, cb)
    want = np.linalg.norm(x.astype(np.float64) @ R.astype(np.float64).T, axis=1)
    off = lambda r: (r.astype(np.float64) - want) / want
    ours, theirs = off(radius.cpu().numpy()), off(chain)
    print(f"radius D{d} {kind}: rms {np.sqrt((ours**2).mean()):.2e} mean {ours.mean():.1e} (chain {np.sqrt((theirs**2).mean()):.2e})")
    assert np.sqrt((ours**2).mean()) <= np.sqrt((theirs**2).mean())
    assert np.abs(ours.mean()) <= 2.0**-25                     # no drift of more than half a rounding


@pytest.mark.parametrize("d,n", [(128, 20_001), (64, 40_001), (128, 4097), (64, 4097), (128, 3)])
def test_compress_of_infinities_nan_and_extreme_vectors(d, n):
    """What the FP32 chain gives, from 4096 vectors on too: an infinity in an input is an infinite radius, not NaN."""
    from polarquant_kv import _ext
    from polarquant_kv import llama_bridge as LB
    rng = np.random.default_rng(d)
    x = rng.standard_normal((n, d)).astype(np.float32)
    special = {0: lambda v: v * np.float32(1e25), 1: lambda v: v * np.float32(0), 2: lambda v: np.where(np.arange(d) == 5, np.inf, v)}
    if n > 3:
        special.update({77: lambda v: np.where(np.arange(d) == d - 1, -np.inf, v), 78: lambda v: np.where(np.arange(d) == 40, np.nan, v),
                        79: lambda v: v * np.float32(1e-20), 80: lambda v: v * np.float32(1e-23), 81: lambda v: v * np.float32(1e-39),
                        200: lambda v: np.full(d, 3.4e38), 4096: lambda v: np.full(d, np.inf), 4095: lambda v: v * np.float32(3e18),
                        300: lambda v: v * np.float32(1e-17)})
    for row, f in special.items():
        x[row] = f(x[row]).astype(np.float32)
    R, cb = orthogonal(d, rng), codebook_for(16, rng)
    radius, packed = LB.compress(torch.from_numpy(x).cuda(), torch.from_numpy(R).cuda(), torch.from_numpy(cb).cuda())
    radius, packed = radius.cpu().numpy(), packed.cpu().numpy()
    want_radius, want_packed = fp32_chain(x, R, cb)
    rows = sorted(special)
    assert np.array_equal(np.isnan(radius), np.isnan(want_radius)) and np.array_equal(np.isinf(radius), np.isinf(want_radius))
    finite = np.isfinite(want_radius)
    # subnormal squares: below 4096 vectors in another order, where a unit in the last place of the sum is up to 2^-10 of it
    np.testing.assert_allclose(radius[finite], want_radius[finite], rtol=2e-6 if n > 3 else 1e-3)
    assert np.array_equal(packed[rows], want_packed[rows])
    assert _ext.poll_device_errors() == 0


@pytest.mark.parametrize("d,n,book", [(128, 20_003, "lloyd"), (64, 40_001, "lloyd"), (128, 4096, "lloyd"), (128, 20_003, "descending"),
                                      (64, 40_001, "descending"), (128, 20_003, "crowded"), (64, 40_001, "pairs"), (128, 20_003, "shuffled"),
                                      (64, 40_001, "eleven"), (64, 40_001, "close"), (128, 20_003, "one")])
def test_near_ties_are_settled_as_an_fp32_chain_does(d, n, book):
    """Half of the coordinates within 1e-6 of a decision point, so that nearly every block goes through the second pass and
    the list of a CTA overflows (512 blocks a tile at D = 128, 256 at D = 64; it holds 480): every stored byte is the
    chain's."""
    from polarquant_kv import _ext
    from polarquant_kv import llama_bridge as LB
    rng = np.random.default_rng(d + n)
    from polarquant_kv.codebook import build_lloyd_max_codebook
    R, cb = orthogonal(d, rng), build_lloyd_max_codebook(d, 4)[0].astype(np.float32)
    points = (cb[1:].astype(np.float64) + cb[:-1]) / 2
    points = points[np.abs(points) < 0.11]
    # tables for the search tree: descending, two decision points in a bucket, levels that occur twice, any order, eleven
    # levels; for the scan: levels closer than 1e-5; one level
    if book == "descending":
        cb = cb[::-1].copy()
    elif book == "crowded":
        cb[8] = cb[7] + np.float32(1e-3)
    elif book == "pairs":
        cb[1::2] = cb[0::2]
    elif book == "shuffled":
        cb = rng.permutation(cb)
    elif book == "eleven":
        cb = rng.permutation(cb[3:14])
    elif book == "close":
        cb[8] = cb[7] + np.float32(2e-6)
    elif book == "one":
        cb = cb[5:6].copy()
    direction = rng.standard_normal((n, d))
    at = rng.permuted(np.tile(np.arange(d) % 2 == 0, (n, 1)), axis=1)
    tied = rng.choice(points, (n, d)) + rng.uniform(-1e-6, 1e-6, (n, d))
    rest = np.where(at, 0.0, direction)
    room = 1.0 - (np.where(at, tied, 0.0) ** 2).sum(1, keepdims=True)
    assert (room > 0).all()
    unit = np.where(at, tied, rest * np.sqrt(room) / np.linalg.norm(rest, axis=1, keepdims=True))
    x = (unit @ R.astype(np.float64) * np.exp(rng.uniform(-5, 5, (n, 1)))).astype(np.float32)
    radius, packed = LB.compress(torch.from_numpy(x).cuda(), torch.from_numpy(R).cuda(), torch.from_numpy(cb).cuda())
    want_radius, want_packed = fp32_chain(x, R, cb)
    differ = int((packed.cpu().numpy() != want_packed).sum())
    assert differ == 0, f"{differ} of {want_packed.size} bytes"
    np.testing.assert_allclose(radius.cpu().numpy(), want_radius, rtol=5e-7)     # two roundings of the radius and its sums
    assert _ext.poll_device_errors() == 0


# the edges of a wave of the kernel with R in shared memory, and buffers off the 16-byte grid, which stay with it
@pytest.mark.parametrize("d,n,offset", [(128, 9472, 0), (128, 9473, 0), (64, 18_944, 0), (64, 18_945, 0), (128, 30_003, 1),
                                        (64, 50_001, 3), (128, 4096, 2)])
def test_compress_kernels_store_the_same_bytes(d, n, offset):
    from polarquant_kv import llama_bridge as LB
    rng = np.random.default_rng(n + offset)
    x, R, cb = kv_like(n, d, rng), orthogonal(d, rng), codebook_for(16, rng)

    def at(a):
        return torch.cat([torch.zeros(offset), torch.from_numpy(a).flatten()]).cuda()[offset:].view(a.shape)

    radius, packed = LB.compress(at(x), at(R), at(cb))
    want_radius, want_packed = fp32_chain(x, R, cb)
    assert np.array_equal(packed.cpu().numpy(), want_packed)
    np.testing.assert_allclose(radius.cpu().numpy(), want_radius, rtol=5e-7)
    first, _ = LB.compress(at(x[:5000]), at(R), at(cb))
    np.testing.assert_allclose(radius[:5000].cpu().numpy(), first.cpu().numpy(), rtol=5e-7)


@pytest.mark.parametrize("d", [128, 96])
def test_attention_on_several_streams_and_in_graphs(d):
    """Sliced calls of different shapes in flight on three streams at once, two of them replayed from CUDA graphs, give what
    they give one after another: no workspace is shared between them."""
    from polarquant_kv import llama_bridge as LB
    rng = np.random.default_rng(d)
    cb = torch.from_numpy(codebook_for(16, rng)).cuda()
    calls, want = [], []
    for hq, hkv, s in ((32, 8, 20_000), (8, 1, 9001), (16, 2, 33_333)):
        pk, kr = (torch.from_numpy(a).cuda() for a in random_cache(hkv, s, d, 16, rng))
        pv, vr = (torch.from_numpy(a).cuda() for a in random_cache(hkv, s, d, 16, rng))
        q = torch.from_numpy(rng.standard_normal((hq, d)).astype(np.float32)).cuda()
        calls.append((q, pk, kr, pv, vr, cb, 0.1))
        want.append(LB.fused_attention(*calls[-1]).clone())
        given = torch.empty_like(q)
        assert LB.fused_attention(*calls[-1], out=given) is given and torch.equal(given, want[-1])
    streams = [torch.cuda.Stream() for _ in calls]
    graphs, outs = [], []
    torch.cuda.synchronize()
    for call, stream in list(zip(calls, streams))[:2]:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            outs.append([LB.fused_attention(*call) for _ in range(2)])
        graphs.append(graph)
    results = []
    for _ in range(30):
        for graph, stream in zip(graphs, streams):
            with torch.cuda.stream(stream):
                graph.replay()
        with torch.cuda.stream(streams[2]):
            results.append(LB.fused_attention(*calls[2]))
    torch.cuda.synchronize()
    assert all(torch.equal(r, want[2]) for r in results)
    for got, ref in zip(outs, want):
        assert all(torch.equal(o, ref) for o in got)


def test_attention_with_a_small_workspace_of_the_callers():
    """Fewer bytes than a call could use: it is sliced less; the counters are zero again afterwards."""
    import ctypes

    from polarquant_kv import _ext
    lib, rng, hq, hkv, s, d = _ext.lib(), np.random.default_rng(1), 8, 2, 9000, 128
    cb = codebook_for(16, rng)
    pk, kr = random_cache(hkv, s, d, 16, rng)
    pv, vr = random_cache(hkv, s, d, 16, rng)
    q = rng.standard_normal((hq, d)).astype(np.float32)
    want = LO.fused_attention(q, pk, kr, pv, vr, cb, 16, 0.1)
    t = [torch.from_numpy(a).cuda() for a in (q, pk, kr, pv, vr, cb)]
    need = lib.polarquant_fused_attention_ws_bytes_c(hq, hkv, s, d)
    assert need > 65536 and lib.polarquant_fused_attention_ws_bytes_c(hq, hkv, 20, d) == 0
    for size in (need, 65536 + 3 * hq * (d + 2) * 4, 65536, 16):
        ws = torch.cat([torch.zeros(65536, dtype=torch.uint8), torch.full((need,), 255, dtype=torch.uint8)]).cuda()
        out = torch.empty(hq, d, device="cuda")
        lib.polarquant_fused_attention_ws_cuda_c(*[x.data_ptr() for x in t], out.data_ptr(), hq, hkv, s, d, 16, ctypes.c_float(0.1),
                                                 ws.data_ptr(), size, torch.cuda.current_stream().cuda_stream)
        assert lib.polarquant_last_error_c() == 0
        assert np.abs(out.cpu().numpy() - want).max() <= 1e-4 * max(1.0, np.abs(want).max())
        assert not ws[:65536].any() and (ws[max(size, 65536):] == 255).all()


@pytest.mark.parametrize("d,s,scale", [(64, 9000, 0.125), (128, 9000, 0.088388346), (64, 700, 0.125), (128, 5000, -0.05), (64, 300, 0.0)])
def test_fused_attention_error_of_large_scores(d, s, scale):
    """Scores of tens: their float32 dot products and one rounding by the radius (a few 2^-24 of a score of 30 or so) are what
    the weights inherit.  The bounds are twice the errors measured.  A negative scale and zero are scales too."""
    from polarquant_kv import _ext
    from polarquant_kv import llama_bridge as LB
    from polarquant_kv.codebook import build_lloyd_max_codebook
    hq, hkv = 32, 8
    rng = np.random.default_rng(d + s)
    cb = build_lloyd_max_codebook(d, 4)[0].astype(np.float32)
    pk, pv = (random_cache(hkv, s, d, 16, rng)[0] for _ in range(2))
    kr, vr = ((30 * (1 + 0.2 * rng.standard_normal((hkv, s)))).astype(np.float32) for _ in range(2))
    q = rng.standard_normal((hq, d)).astype(np.float32)
    dev = lambda a: torch.from_numpy(a).cuda()
    out = LB.fused_attention(dev(q), dev(pk), dev(kr), dev(pv), dev(vr), dev(cb), scale).cpu().numpy()
    want = LO.fused_attention(q, pk, kr, pv, vr, cb, 16, float(np.float32(scale)))
    off = np.linalg.norm(out - want, axis=1) / np.linalg.norm(want, axis=1)
    print(f"attention D{d} s={s} scale {scale}: relative error per head, geometric mean {np.exp(np.log(off).mean()):.2e}")
    assert np.exp(np.log(off).mean()) <= 1e-6 and off.max() <= 5e-6
    assert _ext.poll_device_errors() == 0


# both kernels of the inverse rotation: few rows (columns and k dealt out), many rows, and in place
@pytest.mark.parametrize("d", [2, 64, 66, 128, 130, 256, 1000])
@pytest.mark.parametrize("rows", [1, 197, 198, 400])
def test_inverse_rotation_kernels_vs_oracle(d, rows):
    from polarquant_kv import _ext
    from polarquant_kv import llama_bridge as LB
    rng = np.random.default_rng(d + rows)
    y, R = rng.standard_normal((rows, d)).astype(np.float32), orthogonal(d, rng)
    yt, Rt = torch.from_numpy(y).cuda(), torch.from_numpy(R).cuda()
    want = LO.inverse_rotate(y, R)
    # chains of up to 1000 float32 multiply-adds of terms below 4 |R|: a few 2^-24 of the row's norm
    bound = 4e-7 * np.linalg.norm(y, axis=1).max()
    assert np.abs(LB.inverse_rotate(yt, Rt).cpu().numpy() - want).max() <= bound
    _ext.lib().polarquant_inverse_rotate_cuda_c(yt.data_ptr(), Rt.data_ptr(), yt.data_ptr(), rows, d, torch.cuda.current_stream().cuda_stream)
    assert np.abs(yt.cpu().numpy() - want).max() <= bound and _ext.lib().polarquant_last_error_c() == 0
