"""Kernels that are chosen by size, at the sizes where they can go wrong: edges of tiles and stages, remainders, the
smallest and the largest of a range. Against plain float64 / integer restatements."""
import numpy as np
import pytest

from litert_b200 import workloads

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def ops():
    from litert_b200 import ops as o

    return o


@pytest.fixture(scope="module")
def ws(ops):
    return ops.Workspace("cuda", 64 << 20)


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _attention(q, k, v, length, scale, cap, mask=None):
    """One row in float64: q [n, h]; k, v [s, nkv, h]."""
    n, h = q.shape
    nkv = k.shape[1]
    out = np.zeros((n, h))
    if length <= 0:
        return out
    for i in range(n):
        kv = i // (n // nkv)
        logit = k[:length, kv].astype(np.float64) @ q[i].astype(np.float64) * scale
        if cap:
            logit = cap * np.tanh(logit / cap)
        if mask is not None:
            logit = logit + mask[:length]
        p = np.exp(logit - logit.max())
        out[i] = p @ v[:length, kv].astype(np.float64) / p.sum()
    return out


@pytest.mark.parametrize("kv", ["f16", "i8", "f32"])
@pytest.mark.parametrize("n,nkv,h", [(8, 1, 256), (6, 2, 128), (4, 4, 64), (3, 1, 64)])
def test_sdpa_decode_over_unequal_pieces(ops, ws, kv, n, nkv, h):
    """The cached tokens of all sequences are cut into equal pieces: lengths that end on and next to units (16 tokens),
    stages (32 to 128) and pieces, empty sequences first, between and last, and rows behind a sequence's last token
    that hold NaN. Bound: keys, queries, values and weights are fp16 operands (2^-11 each), fp16 outputs another 2^-11:
    five roundings of 4.9e-4 at most."""
    rng = np.random.default_rng(n * 100 + h)
    s_max = 1001
    lengths = np.asarray([0, 1, 15, 16, 17, 0, 31, 63, 64, 65, 127, 128, 129, 255, 640, 1000, 1001, 0], np.int32)
    b = len(lengths)
    q = rng.standard_normal((b, 1, n, h)).astype(np.float32)
    k = rng.standard_normal((b, s_max, nkv, h)).astype(np.float32)
    v = rng.standard_normal((b, s_max, nkv, h)).astype(np.float32)
    kw = dict(scale=1.0 / np.sqrt(h), logit_cap=30.0 if h == 128 else 0.0)
    mask = None
    if kv == "i8":
        kd, ks = workloads.quantize_kv_per_token(k)
        vd, vs = workloads.quantize_kv_per_token(v)
        kf, vf = kd.astype(np.float32) * ks[..., None], vd.astype(np.float32) * vs[..., None]
        kw.update(k_scale=dev(ks), v_scale=dev(vs))
    else:
        t = np.float16 if kv == "f16" else np.float32
        kd, vd = k.astype(t), v.astype(t)
        kf, vf = kd.astype(np.float32), vd.astype(np.float32)
        for i, length in enumerate(lengths):
            kd[i, length:] = np.nan
            vd[i, length:] = np.nan
    if kv == "f32":
        mask = rng.standard_normal((b, s_max)).astype(np.float32)
        kw["mask"] = dev(mask)
    else:
        q = q.astype(np.float16)
    out = ops.sdpa_decode(dev(q), dev(kd), dev(vd), lengths=dev(lengths), ws=ws, **kw).float().cpu().numpy()
    ws.check_status()
    for i, length in enumerate(lengths):
        want = _attention(q[i, 0].astype(np.float32), kf[i], vf[i], int(length), kw["scale"], kw["logit_cap"],
                          None if mask is None else mask[i])
        assert np.max(np.abs(out[i, 0] - want)) <= 5 * 2.0 ** -11 * max(np.max(np.abs(want)), 1e-30), (i, length)


@pytest.mark.parametrize("b,s_max,kv", [(1, 5000, "f16"), (1, 63, "i8"), (2, 8192, "i8"), (70, 40, "f16")])
def test_sdpa_decode_with_many_records_per_sequence_and_many_sequences(ops, ws, b, s_max, kv):
    """One sequence over all SMs (over 64 records to merge), one piece in all, and more sequences than a warp has lanes."""
    rng = np.random.default_rng(b + s_max)
    n, nkv, h = 8, 1, 128
    q = rng.standard_normal((b, 1, n, h)).astype(np.float16)
    k = rng.standard_normal((b, s_max, nkv, h)).astype(np.float16)
    v = rng.standard_normal((b, s_max, nkv, h)).astype(np.float16)
    lengths = rng.integers(s_max // 2, s_max + 1, b).astype(np.int32)
    kw = {}
    kd, vd, kf, vf = k, v, k.astype(np.float32), v.astype(np.float32)
    if kv == "i8":
        kd, ks = workloads.quantize_kv_per_token(k)
        vd, vs = workloads.quantize_kv_per_token(v)
        kf, vf = kd.astype(np.float32) * ks[..., None], vd.astype(np.float32) * vs[..., None]
        kw = dict(k_scale=dev(ks), v_scale=dev(vs))
    out = ops.sdpa_decode(dev(q), dev(kd), dev(vd), lengths=dev(lengths), ws=ws, **kw).float().cpu().numpy()
    for i in range(b):
        want = _attention(q[i, 0].astype(np.float32), kf[i], vf[i], int(lengths[i]), 1.0 / np.sqrt(h), 0.0)
        assert np.max(np.abs(out[i, 0] - want)) <= 5 * 2.0 ** -11 * np.max(np.abs(want)), i


@pytest.mark.parametrize("kv", ["f16", "i8"])
@pytest.mark.parametrize("n,nkv,h,s_max", [(8, 1, 256, 1100), (7, 1, 128, 700), (6, 2, 64, 130), (4, 4, 256, 64)])
def test_sdpa_rows_of_any_lengths(ops, kv, n, nkv, h, s_max):
    """Query tokens that share one cache, in no order of their lengths: limits on and next to tiles (64 tokens) and
    chunks (256, 320), empty rows, a last CTA that is not full, and cached values that are not finite behind some rows'
    limits. Bound as for the decode step: five roundings of 2^-11."""
    _check_rows(ops, kv, n, nkv, h, s_max, 83)


def _check_rows(ops, kv, n, nkv, h, s_max, more):
    rng = np.random.default_rng(n * 100 + h)
    marks = [0, 1, 63, 64, 65, 127, 128, 129, 255, 256, 257, 319, 320, 321, 640, 1024, s_max - 1, s_max]
    lengths = np.asarray([m for m in marks if m <= s_max] + list(rng.integers(1, s_max + 1, more)), np.int32)
    rng.shuffle(lengths)
    rows = len(lengths)
    q = rng.standard_normal((rows, n, h)).astype(np.float16)
    k = rng.standard_normal((s_max, nkv, h)).astype(np.float16)
    v = rng.standard_normal((s_max, nkv, h)).astype(np.float16)
    kw = dict(scale=1.0 / np.sqrt(h), logit_cap=30.0 if h == 128 else 0.0)
    bad = s_max
    if kv == "i8":
        kd, ks = (a[0] for a in workloads.quantize_kv_per_token(k[None]))
        vd, vs = (a[0] for a in workloads.quantize_kv_per_token(v[None]))
        kf, vf = kd.astype(np.float32) * ks[..., None], vd.astype(np.float32) * vs[..., None]
        kw.update(k_scale=dev(ks), v_scale=dev(vs))
    else:
        bad = s_max * 3 // 4 + 5  # a token whose value is not finite
        v[bad, :, ::3] = np.inf
        kd, vd, kf, vf = k, v, k.astype(np.float32), v.astype(np.float32)
    out = ops.sdpa_rows(dev(q), dev(kd), dev(vd), dev(lengths), **kw).float().cpu().numpy()
    for i, length in enumerate(lengths):
        if length > bad:
            assert not np.isfinite(out[i, :, ::3]).any() and np.isfinite(out[i, :, 1::3]).all()
            continue
        want = _attention(q[i].astype(np.float32), kf, vf, int(length), kw["scale"], kw["logit_cap"])
        assert np.max(np.abs(out[i] - want)) <= 5 * 2.0 ** -11 * max(np.max(np.abs(want)), 1e-30), (i, length)


@pytest.mark.parametrize("kv", ["f16", "i8"])
@pytest.mark.parametrize("n,nkv,h,s_max", [(8, 1, 256, 1100), (7, 1, 128, 700), (6, 2, 64, 330), (4, 4, 256, 164)])
@pytest.mark.parametrize("above", [0, 1])
def test_sdpa_rows_on_both_sides_of_their_rule(ops, kv, n, nkv, h, s_max, above):
    """More than 262144 (row, cached token, KV head) triples run 64 (row, head) pairs to a CTA, others a warp per row:
    the lengths and values of the test above, one row fewer and one more."""
    marks = sum(m <= s_max for m in [0, 1, 63, 64, 65, 127, 128, 129, 255, 256, 257, 319, 320, 321, 640, 1024, s_max - 1, s_max])
    _check_rows(ops, kv, n, nkv, h, s_max, 262144 // (s_max * nkv) + above - marks)


@pytest.mark.parametrize("d", [4, 1000, 1024, 1028, 2048, 2052, 4096])
def test_norm_of_many_rows_equals_that_of_a_few(ops, d):
    """33 rows and more are kept in registers, four neighbours per thread: widths on and next to a thread's pieces.
    Residuals are equal; the sum of squares is added in another order (relative error up to d 2^-24), so a scale may
    differ by that and an integer by one where a value lies on a rounding boundary."""
    rng = np.random.default_rng(d)
    h = rng.standard_normal((40, d)).astype(np.float32) * 3
    delta, gain = rng.standard_normal((40, d)).astype(np.float32), rng.uniform(0.9, 1.1, d).astype(np.float32)
    many = dev(h)
    got = ops.add_rmsnorm_quantize(many, dev(delta), dev(gain))
    for r in range(0, 40, 20):
        few = dev(h[r:r + 20])
        want = ops.add_rmsnorm_quantize(few, dev(delta[r:r + 20]), dev(gain))
        assert torch.equal(few, many[r:r + 20])
        assert torch.allclose(got.scales[r:r + 20], want.scales[:20], rtol=d * 2.0 ** -24, atol=0)
        assert torch.equal(got.zero_points[r:r + 20], want.zero_points[:20])
        diff = (got.rows()[r:r + 20].int() - want.rows()[:20].int()).abs()
        assert int(diff.max()) <= 1 and float((diff != 0).float().mean()) <= 1e-3


@pytest.mark.parametrize("kv", ["f16", "i8"])
@pytest.mark.parametrize("heads,kv_heads,h", [(8, 1, 256), (6, 2, 128), (3, 3, 128)])
def test_rotation_of_many_rows_equals_that_of_a_few(ops, kv, heads, kv_heads, h):
    """33 rows and more take a warp per (row, head): the same bits as a block per (row, head)."""
    rng = np.random.default_rng(heads)
    rows, max_seq = 45, 50
    qkv = rng.standard_normal((rows, (heads + 2 * kv_heads) * h)).astype(np.float32)
    pos = (np.arange(rows) + 8).astype(np.int32)  # the last three lie past the cache
    table = ops.rope_table(max_seq + 1, h)
    out = []
    for pieces in ((0, rows), (0, 25, rows)):
        kc = torch.zeros((1, max_seq, kv_heads, h), dtype=torch.float16 if kv == "f16" else torch.int8, device="cuda")
        vc = torch.zeros_like(kc)
        ks = torch.zeros((1, max_seq, kv_heads), device="cuda") if kv == "i8" else None
        vs = torch.zeros_like(ks) if kv == "i8" else None
        q = [ops.rope_kv_append(dev(qkv[a:b]), heads, kv_heads, h, table, dev(pos[a:b]), kc, vc, ks, vs, one_sequence=True)
             for a, b in zip(pieces, pieces[1:])]
        out.append([torch.cat(q), kc, vc] + ([ks, vs] if kv == "i8" else []))
    assert all(torch.equal(a, b) for a, b in zip(*out))


def _decode_case(rng, lengths, s_max, n, nkv, h):
    """Queries that fp16 holds exactly, int8 keys with scales: the logits of float32 arithmetic over exact operands."""
    b = len(lengths)
    q = rng.standard_normal((b, 1, n, h)).astype(np.float16).astype(np.float32)
    k8 = rng.integers(-127, 128, (b, s_max, nkv, h)).astype(np.int8)
    ks = rng.uniform(0.005, 0.02, (b, s_max, nkv)).astype(np.float32)
    return q, k8, ks


@pytest.mark.parametrize("scales", ["small", "growing", "shrinking", "zeros among them", "large"])
@pytest.mark.parametrize("n,nkv,h", [(8, 1, 256), (6, 2, 128), (4, 4, 64)])
def test_sdpa_decode_int8_value_scales_of_any_size(ops, ws, scales, n, nkv, h):
    """Softmax weights times value scales are fp16 operands: scales far below and above what fp16 holds, and such that
    change along the cache, cost no more than those near one (caches over 2048 tokens: the split kernel). Bound: an fp16 rounding (2^-11) of each weight, and half
    the smallest fp16 step (2^-25) of the largest scale, which is counted in units of at most twice itself."""
    rng = np.random.default_rng(h)
    s_max, lengths = 2100, np.asarray([2100, 0, 700, 33, 1], np.int32)
    b = len(lengths)
    q, k8, ks = _decode_case(rng, lengths, s_max, n, nkv, h)
    v8 = rng.integers(-127, 128, (b, s_max, nkv, h)).astype(np.int8)
    vs = rng.uniform(0.5, 1.0, (b, s_max, nkv))
    steps = np.linspace(-9, 3, s_max)[None, :, None]
    vs = {"small": vs * 1e-6, "growing": vs * 10.0 ** steps, "shrinking": vs * 10.0 ** -steps,
          "zeros among them": vs * 1e-4 * (rng.random(vs.shape) < 0.5), "large": vs * 1e6}[scales].astype(np.float32)
    out = ops.sdpa_decode(dev(q), dev(k8), dev(v8), lengths=dev(lengths), k_scale=dev(ks), v_scale=dev(vs), ws=ws)
    out = out.cpu().numpy()
    kf, vf = k8.astype(np.float64) * ks[..., None], v8.astype(np.float64) * vs[..., None]
    for i, length in enumerate(lengths):
        if length == 0:
            assert not out[i].any()
            continue
        want = _attention(q[i, 0], kf[i], vf[i], int(length), 1.0 / np.sqrt(h), 0.0)
        size = _attention(q[i, 0], kf[i], np.abs(vf[i]), int(length), 1.0 / np.sqrt(h), 0.0)
        top = np.repeat(vs[i, :length].max(0), n // nkv)[:, None] * 127.0
        assert np.all(np.abs(out[i, 0] - want) <= 1.05 * 2.0 ** -11 * size + 2.0 ** -24 * top), i


@pytest.mark.parametrize("kv", ["f16", "f32"])
@pytest.mark.parametrize("n,nkv,h", [(8, 1, 256), (6, 2, 128), (4, 4, 64)])
def test_sdpa_decode_weights_are_not_rounded_to_fp16(ops, ws, kv, n, nkv, h):
    """float16 and float32 rows in the split kernel: a weight is the sum of two fp16 operands (2^-22 of it is lost), so that with operands
    fp16 holds and float32 outputs only float32 arithmetic is left: 2h products per logit of a few units at 2^-23
    each, taken as 2^-15 of the output. A single fp16 weight is 2^-12 off, 1.8e-4 here."""
    rng = np.random.default_rng(h)
    s_max, lengths = 2100, np.asarray([2100, 64, 333], np.int32)
    b = len(lengths)
    half = lambda a: a.astype(np.float16).astype(np.float32)
    q = half(rng.standard_normal((b, 1, n, h)))
    k, v = half(rng.standard_normal((b, s_max, nkv, h))), half(rng.standard_normal((b, s_max, nkv, h)))
    t = np.float16 if kv == "f16" else np.float32
    out = ops.sdpa_decode(dev(q), dev(k.astype(t)), dev(v.astype(t)), lengths=dev(lengths), ws=ws).cpu().numpy()
    for i, length in enumerate(lengths):
        want = _attention(q[i, 0], k[i], v[i], int(length), 1.0 / np.sqrt(h), 0.0)
        assert np.linalg.norm(out[i, 0] - want) <= 2.0 ** -15 * np.linalg.norm(want), i


def _at_offset(a, nbytes):
    """The array on the device, `nbytes` behind a 256-byte boundary."""
    flat = torch.from_numpy(np.ascontiguousarray(a)).cuda().reshape(-1)
    raw = torch.empty(flat.numel() * flat.element_size() + 256, dtype=torch.uint8, device="cuda")
    at = raw[nbytes:nbytes + flat.numel() * flat.element_size()].view(flat.dtype).reshape(a.shape)
    at.copy_(flat.reshape(a.shape))
    assert at.data_ptr() % 256 == nbytes
    return at


@pytest.mark.parametrize("s_max,b", [(700, 5), (60000, 1)])
@pytest.mark.parametrize("n,nkv,h", [(8, 1, 256), (6, 2, 128), (4, 4, 64)])
def test_sdpa_decode_int8_cache_on_an_8_byte_boundary(ops, ws, s_max, b, n, nkv, h):
    """Copies by the TMA need 16 bytes; a cache on 8 is taken by the kernel that loads rows straight, whatever its
    length. Also quantized. Bound: fp16 weights, queries and outputs, as for the other decode tests."""
    rng = np.random.default_rng(h + b)
    lengths = np.asarray([s_max, 0, 1, 65, 640][:b], np.int32)
    q = rng.standard_normal((b, 1, n, h)).astype(np.float16)
    kd = rng.integers(-127, 128, (b, s_max, nkv, h)).astype(np.int8)
    vd = rng.integers(-127, 128, (b, s_max, nkv, h)).astype(np.int8)
    ks, vs = (rng.uniform(0.005, 0.02, (b, s_max, nkv)).astype(np.float32) for _ in range(2))
    k, v = _at_offset(kd, 8), _at_offset(vd, 8)
    out = ops.sdpa_decode(dev(q), k, v, lengths=dev(lengths), k_scale=dev(ks), v_scale=dev(vs), ws=ws).float().cpu().numpy()
    rows = ops.sdpa_decode_quantized(dev(q.astype(np.float32)), k, v, dev(lengths), k_scale=dev(ks), v_scale=dev(vs))
    scale, zp = rows.scales[:b].cpu().numpy(), rows.zero_points[:b].cpu().numpy()
    quant = (rows.rows().cpu().numpy().astype(np.float64) - zp[:, None]) * scale[:, None]
    for i, length in enumerate(lengths):
        want = _attention(q[i, 0].astype(np.float32), kd[i].astype(np.float32) * ks[i][..., None],
                          vd[i].astype(np.float32) * vs[i][..., None], int(length), 1.0 / np.sqrt(h), 0.0)
        bound = 5 * 2.0 ** -11 * max(np.max(np.abs(want)), 1e-30)
        assert np.max(np.abs(out[i, 0] - want)) <= bound, i
        assert np.max(np.abs(quant[i].reshape(n, h) - want)) <= bound + 0.51 * scale[i], i


@pytest.mark.parametrize("kv", ["f16", "i8", "f32"])
def test_sdpa_decode_workspace_on_a_4_byte_boundary(ops, kv):
    """The records move up to the next boundary: same bits as with an aligned workspace, nothing written outside."""
    import ctypes

    from litert_b200 import _lib

    rng = np.random.default_rng(5)
    b, s_max, n, nkv, h = 3, 3000, 8, 2, 128
    q = dev(rng.standard_normal((b, 1, n, h)).astype(np.float32))
    x = [rng.standard_normal((b, s_max, nkv, h)) for _ in range(2)]
    kw = {}
    if kv == "i8":
        kv_t = [dev(np.clip(np.rint(a * 40), -127, 127).astype(np.int8)) for a in x]
        kw = {a: torch.full((b, s_max, nkv), 0.02, device="cuda") for a in ("k_scale", "v_scale")}
    else:
        kv_t = [dev(a.astype(np.float16 if kv == "f16" else np.float32)) for a in x]
    lib = _lib.load()
    need = lib.b200_sdpa_workspace_bytes(b, n, nkv, h, s_max)
    guard = torch.full((need + 512,), 0x5A, dtype=torch.uint8, device="cuda")
    out = torch.empty_like(q)
    p = lambda t: None if t is None else ctypes.c_void_p(t.data_ptr())
    _lib.check(lib.b200_sdpa_decode(p(q), p(kv_t[0]), p(kv_t[1]), p(kw.get("k_scale")), p(kw.get("v_scale")), None, None,
                                    p(out), b, n, nkv, h, s_max, 2, {"f16": 0, "i8": 1, "f32": 2}[kv], 0.0, 0.0,
                                    ctypes.c_void_p(guard.data_ptr() + 260), need, None))
    torch.cuda.synchronize()
    assert torch.equal(out, ops.sdpa_decode(q, *kv_t, ws=ops.Workspace("cuda"), **kw))
    g = guard.cpu().numpy()
    assert (g[:260] == 0x5A).all() and (g[260 + need:] == 0x5A).all()


def test_sdpa_decode_says_what_it_does_not_take(ops, ws):
    """fp16 rows on an 8-byte boundary run on the fallback, which holds all logits in shared memory."""
    from litert_b200._lib import B200Error

    q = torch.randn((1, 1, 8, 64), device="cuda")
    mk = lambda s: _at_offset(np.zeros((1, s, 1, 64), np.float16), 8)
    assert not ops.sdpa_decode(q, mk(300), mk(300), ws=ws).any()
    with pytest.raises(B200Error, match="alignment"):
        ops.sdpa_decode(q, mk(60000), mk(60000), ws=ws)


@pytest.mark.parametrize("kv", ["f16", "i8", "f32"])
@pytest.mark.parametrize("b,n,nkv,h,s_max", [(1, 8, 1, 128, 8192), (1, 8, 1, 128, 8193), (2, 8, 8, 64, 1024),
                                             (2, 8, 8, 64, 1025), (1, 8, 4, 64, 2048), (1, 8, 4, 64, 2049),
                                             (3, 8, 1, 256, 1023), (3, 8, 1, 256, 1024), (3, 8, 1, 256, 1025),
                                             (9, 8, 8, 64, 2100), (70, 4, 1, 128, 40), (64, 4, 1, 256, 256), (65, 4, 1, 256, 256),
                                             (65, 4, 1, 256, 257), (33, 4, 2, 128, 512), (33, 4, 2, 128, 513)])
def test_sdpa_decode_on_both_sides_of_its_rules(ops, ws, kv, b, n, nkv, h, s_max):
    """Sizes next to those where another kernel, or another shortest piece, is taken, lengths from nothing to all of the
    cache. Bound: as for the kernels' other tests, five roundings of 2^-11."""
    rng = np.random.default_rng(b * s_max)
    lengths = rng.integers(0, s_max + 1, b).astype(np.int32)
    lengths[0] = s_max
    q = rng.standard_normal((b, 1, n, h)).astype(np.float32 if kv == "f32" else np.float16)
    k, v = (rng.standard_normal((b, s_max, nkv, h)).astype(np.float32) for _ in range(2))
    kw = {}
    if kv == "i8":
        kd, ks = workloads.quantize_kv_per_token(k)
        vd, vs = workloads.quantize_kv_per_token(v)
        k, v = kd.astype(np.float32) * ks[..., None], vd.astype(np.float32) * vs[..., None]
        kw = dict(k_scale=dev(ks), v_scale=dev(vs))
    else:
        kd, vd = (a.astype(np.float16 if kv == "f16" else np.float32) for a in (k, v))
        k, v = kd.astype(np.float32), vd.astype(np.float32)
    out = ops.sdpa_decode(dev(q), dev(kd), dev(vd), lengths=dev(lengths), ws=ws, **kw).float().cpu().numpy()
    for i, length in enumerate(lengths):
        want = _attention(q[i, 0].astype(np.float32), k[i], v[i], int(length), 1.0 / np.sqrt(h), 0.0)
        assert np.max(np.abs(out[i, 0] - want)) <= 5 * 2.0 ** -11 * max(np.max(np.abs(want)), 1e-30), (i, length)


_FC_SHAPES = [
    # cluster kernel: one or two columns and four at a time, one pass and several, partial passes and n tiles
    (2, 300, 2048), (3, 300, 2048), (17, 4096, 2048), (32, 1000, 3000), (33, 1000, 3000), (64, 2048, 2048), (32, 11000, 512),
    (300, 200, 1024), (257, 700, 4300), (66, 900, 2048),
    # persistent kernel, 64 rows per pass: whole reductions and cut ones
    (66, 1000, 1024), (129, 2000, 700), (128, 6000, 4200), (400, 1300, 4500), (300, 1300, 8300), (90, 2500, 16384),
    # 128 rows per pass
    (130, 4097, 1500), (100, 9000, 600), (700, 2000, 300), (150, 2500, 8200), (513, 2100, 5000),
    # 256 rows per pass
    (250, 4001, 4096), (200, 8200, 1000), (513, 3001, 2100), (1000, 300, 6000), (512, 1000, 4500)]


@pytest.mark.parametrize("m,n,k", _FC_SHAPES)
def test_fully_connected_by_every_route(ops, ws, oracle, m, n, k):
    """Shapes that the rules on rows, tiles and reduction length send to each kernel and pass size. Bit-equal to the
    oracle for the rows next to edges of passes and some others (a row's result does not depend on the other rows)."""
    rng = np.random.default_rng(m + n + k)
    rows = sorted({r for e in range(0, m + 64, 64) for r in (e - 1, e) if 0 <= r < m} | {m - 1} | set(rng.integers(0, m, 4).tolist()))
    w = rng.integers(-127, 128, (n, k)).astype(np.int8)
    scales = rng.uniform(1e-3, 1e-2, n).astype(np.float32)
    packed = ops.PackedInt8Weights(dev(w))
    x = rng.standard_normal((m, k)).astype(np.float32)
    y = ops.fully_connected_hybrid(dev(x), packed, dev(scales), ws=ws).cpu().numpy()
    assert np.array_equal(y[rows], oracle.fc_hybrid(x[rows], w, scales))
    xq = rng.integers(-128, 128, (m, k)).astype(np.int8)
    bias = rng.integers(-5000, 5001, n).astype(np.int32)
    out_scale = float(np.float32(0.02 * 5.5e-3 * 74 * np.sqrt(k)))
    mult, shift = oracle.fc_per_channel_multipliers(0.02, out_scale, scales)
    yq = ops.fully_connected_int8(dev(xq), packed, dev(bias), 3, -5, dev(mult), dev(shift), ws=ws).cpu().numpy()
    assert np.array_equal(yq[rows], oracle.fc_int8_per_channel(xq[rows], w, bias, 3, 0.02, scales, out_scale, -5))
    ws.check_status()


@pytest.mark.parametrize("kv", [np.float16, np.float32])
def test_quantized_attention_takes_float32_queries_only(ops, kv):
    from litert_b200._lib import B200Error

    q = torch.randn((2, 1, 8, 128), device="cuda")
    k = dev(np.zeros((2, 100, 1, 128), kv))
    lengths = torch.tensor([100, 7], dtype=torch.int32, device="cuda")
    assert not ops.sdpa_decode_quantized(q, k, k, lengths).rows().any()
    with pytest.raises(B200Error):
        ops.sdpa_decode_quantized(q.half(), k, k, lengths)
