"""The packed parameter structures of the binding against the ctypes mirrors filled field by field."""
import ctypes as C

import pytest

import brodiffusion_b200 as bd


@pytest.mark.parametrize("cls,pack", [(bd.SdpaParams, bd._pack_sdpa), (bd.QkvProjParams, bd._pack_qkv),
                                      (bd.QkvoParams, bd._pack_qkvo), (bd.NormRopeJob, bd._pack_job)])
def test_packed_parameters_are_the_structure(cls, pack):
    ref, values = cls(), []
    for i, (name, t) in enumerate(cls._fields_):
        n = getattr(t, "_length_", 1)
        v = [0.25 * i if t is C.c_float else 1000 * i + e + 1 for e in range(n)]
        values += v
        if n > 1:
            for e in range(n):
                getattr(ref, name)[e] = v[e]
        else:
            setattr(ref, name, v[0])
    raw = pack(*values)
    got = cls.from_buffer_copy(raw)
    assert len(raw) == C.sizeof(cls)
    for name, t in cls._fields_:
        a, b = getattr(ref, name), getattr(got, name)
        assert list(a) == list(b) if getattr(t, "_length_", 1) > 1 else a == b, name


def test_floats_beyond_fp32_are_infinite():
    for x in (1e300, -1e300, float("inf"), float("nan"), 0.0, 1, 3.4e38, 3.5e38, 1e-50):
        a, b = bd._f32(x), C.c_float(x).value
        assert C.c_float(a).value == b or (b != b and a != a)
        n = [0] * sum(getattr(t, "_length_", 1) for _, t in bd.SdpaParams._fields_)
        n[[name for name, t in bd.SdpaParams._fields_ for _ in range(getattr(t, "_length_", 1))].index("softmax_scale")] = a
        got = bd.SdpaParams.from_buffer_copy(bd._pack_sdpa(*n)).softmax_scale
        assert got == b or (b != b and got != got)


def test_c_functions_take_their_own_structure_only():
    """Through ``lib()``: a structure, its reference or its array; what is something else must not be read as one."""
    L = bd.lib()
    calls = {
        "bdattn_sdpa_fwd": (bd.SdpaParams, lambda p: (p, None)),
        "bdattn_qkvo_fwd": (bd.QkvoParams, lambda p: (p, None)),
        "bdattn_qkvo_fwd_static": (bd.QkvoParams, lambda p: (p, None)),
        "bdattn_qkv_norm_rope_fwd": (bd.QkvProjParams, lambda p: (p, None)),
        "bdattn_rmsnorm_rope": (bd.NormRopeJob, lambda p: (p, 1, bd.BF16, 1, 64, 1e-6, 0, None)),
    }
    for name, (cls, args) in calls.items():
        own, fn = cls(), getattr(L, name)
        for p in (None, own, C.byref(own), C.pointer(own), (cls * 1)()):
            assert fn(*args(p)) == -1            # null or all zeros: refused by the entry point itself
        other = bd.QkvoParams() if cls is not bd.QkvoParams else bd.SdpaParams()
        for p in (other, C.byref(other), bytes(own), b"", 4096, C.c_void_p(4096), "x"):
            with pytest.raises(C.ArgumentError):
                fn(*args(p))


def test_arguments_of_other_types_are_type_errors():
    import torch
    x = torch.zeros(4, 64, dtype=torch.bfloat16)
    w, g = torch.zeros(64, 64, dtype=torch.bfloat16), torch.zeros(64)
    for call in (lambda v: bd.sdpa_fwd(x, x, x, x, 1, num_kv_heads=v), lambda v: bd.sdpa_fwd(x, x, x, x, 1, softmax_scale=v and "1"),
                 lambda v: bd.rmsnorm_rope([dict(x=x, out=x, gain=g, rope_row0=v)], 1, 64),
                 lambda v: bd.qkvo_fwd(x, None, w, w, w, w, None, v, x, None),
                 lambda v: bd.qkv_norm_rope_fwd(x, w, w, w, x, x, x, 1, 64, rope_row0=v)):
        with pytest.raises(TypeError):
            call(2.0)
