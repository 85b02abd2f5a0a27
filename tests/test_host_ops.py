"""The native form of the small calls (csrc/host_ops.cc) against the general path through ctypes: same results, same
refusals, and no call that only one of them takes."""
import warnings

import numpy as np
import pytest
import torch


def test_a_missing_or_unusable_extension_leaves_the_general_path(monkeypatch, tmp_path):
    from litert_b200 import _lib

    absent = tmp_path / "_host_ops.so"
    monkeypatch.setattr(_lib, "host_ops_path", lambda: str(absent))
    host = _lib.host_ops()
    assert host.fc_int8(1, 2) is None and host.fc_hybrid() is None and host.fc_w4() is None and host.sdpa_decode() is None
    absent.write_bytes(b"not a library")
    with pytest.warns(UserWarning, match="does not load"):
        assert _lib.host_ops().sdpa_decode() is None
    monkeypatch.setattr(_lib, "LIB_PATH", str(tmp_path / "liblitert_b200.so"))
    assert _lib.host_ops().fc_w4() is None  # (importing ops does not need the kernels' library)


def test_the_extension_is_named_by_what_it_is_built_for():
    from litert_b200 import _lib

    assert torch.__version__ in _lib.host_ops_path()


@pytest.fixture()
def both(monkeypatch):
    """A call through the extension, and again without it."""
    from litert_b200 import _lib, ops

    native = ops._host
    assert native is not _lib._GeneralPath, "the extension is not built"

    def run(call):
        monkeypatch.setattr(ops, "_host", native)
        a = call()
        monkeypatch.setattr(ops, "_host", _lib._GeneralPath)
        return a, call()

    return run


def _inputs(m=5, n=200, k=320):
    from litert_b200 import ops

    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    w8 = torch.randint(-127, 128, (n, k), generator=g, device="cuda").to(torch.int8)
    w4 = torch.randint(0, 256, (n, k // 2), generator=g, device="cuda").to(torch.uint8)
    return dict(x=torch.randn((m, k), generator=g, device="cuda"), w8=ops.PackedInt8Weights(w8),
                xq=torch.randint(-128, 128, (m, k), generator=g, device="cuda").to(torch.int8),
                w4=ops.PackedInt4Weights(w4, torch.rand((n, k // 32), generator=g, device="cuda").half(), 32),
                scales=torch.rand(n, generator=g, device="cuda"),
                mult=torch.full((n,), 1 << 30, dtype=torch.int32, device="cuda"),
                shift=torch.full((n,), -7, dtype=torch.int32, device="cuda"))


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["plain", "not contiguous", "shifted by one", "three dimensions", "out", "no workspace"])
def test_fully_connected_both_ways(both, form):
    from litert_b200 import ops

    d = _inputs()
    ws = None if form == "no workspace" else ops.Workspace("cuda")

    def arrange(t):
        if form == "not contiguous":
            return torch.stack([t, t], -1)[..., 0]
        if form == "shifted by one":
            flat = torch.empty(t.numel() + 1, dtype=t.dtype, device="cuda")
            flat[1:] = t.reshape(-1)
            return flat[1:].view(t.shape)
        return t.reshape(1, *t.shape) if form == "three dimensions" else t

    x, xq = arrange(d["x"]), arrange(d["xq"])
    out = lambda dtype: torch.empty((5, 200), dtype=dtype, device="cuda") if form == "out" else None
    calls = [lambda o=out(torch.int8): (o, ops.fully_connected_int8(xq, d["w8"], None, -128, 3, d["mult"], d["shift"], ws=ws, out=o)),
             lambda o=out(torch.float32): (o, ops.fully_connected_hybrid(x, d["w8"], d["scales"], ws=ws, out=o)),
             lambda o=out(torch.float32): (o, ops.fully_connected_blockwise4(x, d["w4"], ws=ws, out=o))]
    for call in calls:
        (o1, y1), (o2, y2) = both(lambda: (lambda r: (r[0], r[1].clone() if r[0] is None else r[1]))(call()))
        assert y1.shape == y2.shape == (5, 200) and torch.equal(y1, y2) and y1.any()
        assert o1 is None or (y1 is o1 and y2 is o2)


@pytest.mark.gpu
def test_zero_points_of_any_integer_type(both):
    """Negating a numpy int8 of -128 overflows: the zero points are negated as C integers."""
    from litert_b200 import ops

    d, ws = _inputs(), ops.Workspace("cuda")
    want = ops.fully_connected_int8(d["xq"], d["w8"], None, -128, 3, d["mult"], d["shift"], ws=ws)
    with warnings.catch_warnings():
        warnings.simplefilter("error")
        for zp in (-128, np.int8(-128), np.int64(-128), np.float32(-128), True):
            a, b = both(lambda: ops.fully_connected_int8(d["xq"], d["w8"], None, zp, np.int8(3), d["mult"], d["shift"], ws=ws))
            assert torch.equal(a, b) and (zp is True or torch.equal(a, want))


@pytest.mark.gpu
def test_attention_both_ways_and_what_neither_takes(both):
    from litert_b200 import ops

    q, k = torch.randn((2, 1, 8, 64), device="cuda"), torch.randn((2, 99, 2, 64), device="cuda")
    lengths = torch.tensor([99, 40], dtype=torch.int32, device="cuda")
    for ws in (None, ops.Workspace("cuda")):
        for scale in (None, 0, 0.3, np.float32(0.3)):
            a, b = both(lambda: ops.sdpa_decode(q, k, k, lengths=lengths, scale=scale, logit_cap=20, ws=ws))
            assert torch.equal(a, b)
        a, b = both(lambda: ops.sdpa_decode(q, k.transpose(0, 1).contiguous().transpose(0, 1), k, ws=ws))
        assert torch.equal(a, b)

    def refused():
        with pytest.raises(TypeError):
            ops.sdpa_decode(q, k, k, logit_cap=None, ws=ops.Workspace("cuda") if warmed is None else warmed)

    warmed = ops.Workspace("cuda")
    ops.sdpa_decode(q, k, k, ws=warmed)  # (its workspace is there: the extension would take the call)
    both(refused)
