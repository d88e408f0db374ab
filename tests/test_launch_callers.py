"""The native callers of the kernels' entry points on the CPU: a ctypes callback stands in for an entry point."""
import ctypes
import os
import threading
import time

import pytest
import torch

from aien_sovereign_core_mv_b200 import kernels as K
from aien_sovereign_core_mv_b200.csrc import build
from aien_sovereign_core_mv_b200.csrc.signatures import SIGNATURES

TYPES = {"P": ctypes.c_void_p, "I": ctypes.c_int, "L": ctypes.c_long, "Z": ctypes.c_size_t, "F": ctypes.c_float, "D": ctypes.c_double}


def bound(types, rc=0):
    """(caller, the list that its calls land in, what must stay alive)"""
    seen = []
    back = ctypes.CFUNCTYPE(ctypes.c_int, *[TYPES[t] for t in types])(lambda *a: seen.append(a) or rc)
    return build.load_launch().bind(ctypes.cast(back, ctypes.c_void_p).value, types, "stand_in"), seen, back


@pytest.mark.parametrize("types", sorted(set(SIGNATURES.values()), key=len)[::9] + [max(SIGNATURES.values(), key=len), SIGNATURES["aien_rope_table"]])
def test_arguments_arrive_as_declared(types):
    call, seen, _keep = bound(types, rc=-3)
    values = {"P": 0x7fff12345678, "I": -7, "L": -(1 << 40), "Z": 1 << 41, "F": 0.5, "D": 0.1}
    args = [values[t] + (i if t in "PILZ" else 0) for i, t in enumerate(types)]
    assert call(*args) == -3 and seen == [tuple(args)]
    assert call.__name__ == "stand_in"


def test_what_a_caller_refuses():
    types = SIGNATURES["aien_add_residual"]                    # PPIIZIIP
    call, seen, _keep = bound(types)
    good = [1, None, 2, 3, 4, 5, 6, 0]
    assert call(*good) == 0 and seen == [(1, None, 2, 3, 4, 5, 6, None)]
    for at, bad in ((0, torch.zeros(3)), (0, 1.0), (0, "a"), (2, 1.5), (2, None), (2, torch.zeros(2))):
        with pytest.raises(TypeError):
            call(*(good[:at] + [bad] + good[at + 1:]))
    with pytest.raises(TypeError):
        call(*good[:-1])
    with pytest.raises(ValueError):
        build.load_launch().bind(1, "IPFIPFIPF", "unknown")
    assert len(seen) == 1


def test_the_device_check_names_the_error():
    check = build.load_launch().on_device
    assert check(K.KernelError, None, None) is None
    with pytest.raises(K.KernelError):
        check(K.KernelError, None, torch.zeros(2))
    with pytest.raises(TypeError):
        check(K.KernelError, 3)


def test_strided_is_as_strided():
    strided = build.load_launch().strided
    for dtype in (torch.float32, torch.bfloat16, torch.uint8):
        t = torch.arange(200).to(dtype)
        for shape, strides, at in (((3, 4), (4, 1), 7), ((), (), 199), ((0, 5), (5, 1), 0), ((2, 3, 4), (50, 1, 3), 11), ((200,), (1,), 0)):
            a, b = strided(t, shape, strides, at), t.as_strided(shape, strides, at)
            assert a.dtype == dtype and a.shape == b.shape and a.stride() == b.stride() and a.data_ptr() == b.data_ptr() and torch.equal(a, b)
            assert a.is_contiguous() == b.is_contiguous()
        for shape, strides, at in (((201,), (1,), 0), ((2,), (1,), 199), ((1,), (1,), -1), ((-1,), (1,), 0)):
            with pytest.raises(ValueError):
                strided(t, shape, strides, at)
    v = strided(torch.full((8,), 3.0), (8,), (1,), 0)          # the view keeps the storage
    assert torch.equal(v, torch.full((8,), 3.0))


def test_two_threads_build_the_callers_at_the_same_time(monkeypatch, tmp_path):
    """Neither takes the other's work folder away; the compiler is a stand-in that reads its table at the end too, the second later than the first."""
    monkeypatch.setenv("AIEN_B200_BUILD_DIR", str(tmp_path))
    runs, made, errors = [], [], []

    def compiler(cmds, what, jobs):
        runs.append(what)
        table = os.path.join(cmds[0][cmds[0].index("-I") + 1], "signatures.inc")
        assert os.path.exists(table)
        time.sleep(0.1 if len(runs) == 1 else 0.4)
        assert os.path.exists(table)
        with open(cmds[0][cmds[0].index("-o") + 1], "w") as f:
            f.write(what)

    monkeypatch.setattr(build, "_run_parallel", compiler)
    start = threading.Barrier(2)

    def thread():
        try:
            start.wait(10)
            made.append(build.build_launch(force=True))
        except BaseException as e:                             # noqa: BLE001  (told below)
            errors.append(e)

    threads = [threading.Thread(target=thread) for _ in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join(30)
    assert not errors and len(made) == 2 and made[0] == made[1] and open(made[0]).read() == "launch" and len(runs) == 2
    assert sorted(os.path.basename(p) for p in os.listdir(tmp_path)) == sorted(os.path.basename(made[0]) + e for e in ("", ".stamp"))
