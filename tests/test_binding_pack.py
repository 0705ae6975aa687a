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
