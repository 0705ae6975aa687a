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
