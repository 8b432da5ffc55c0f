"""A context made while a green context is current, i.e. in a process that gives
it a part of the GPU's SMs: the Newton solve's cooperative launch is sized by
that part, not by the device, so a step runs as on the whole GPU.  The block has
more points than the part holds threads at once.  Fewer SMs change where a point
is computed and none of its operations, so two steps give the whole GPU's bits
(which the other RK3 tests compare with the oracle).  In child processes, since
the green context stays current."""
import ctypes as C
import os
import subprocess
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
SMS, UNSUPPORTED = 16, 77


def _green_context(n):
    """Makes a green context of n SMs current; False where the driver has none."""
    cu = C.CDLL("libcuda.so.1")

    def ok(rc, what):
        if rc:
            print("%s: %d" % (what, rc))
        return rc == 0

    # CUdevResource is a plain structure of 144 bytes whose fields the driver fills
    whole, part, rest = ((C.c_uint64 * 64)() for _ in range(3))
    dev, ctx, groups = C.c_int(0), C.c_void_p(), C.c_uint(1)
    desc, green, primary = C.c_void_p(), C.c_void_p(), C.c_void_p()
    return (ok(cu.cuInit(0), "cuInit") and ok(cu.cuDeviceGet(C.byref(dev), 0), "cuDeviceGet") and
            ok(cu.cuDevicePrimaryCtxRetain(C.byref(primary), dev), "cuDevicePrimaryCtxRetain") and
            ok(cu.cuDeviceGetDevResource(dev, whole, 1), "cuDeviceGetDevResource") and
            ok(cu.cuDevSmResourceSplitByCount(part, C.byref(groups), whole, rest, 0, C.c_uint(n)), "cuDevSmResourceSplitByCount") and
            ok(cu.cuDevResourceGenerateDesc(C.byref(desc), part, 1), "cuDevResourceGenerateDesc") and
            ok(cu.cuGreenCtxCreate(C.byref(green), desc, dev, 1), "cuGreenCtxCreate") and
            ok(cu.cuCtxFromGreenCtx(C.byref(ctx), green), "cuCtxFromGreenCtx") and
            ok(cu.cuCtxSetCurrent(ctx), "cuCtxSetCurrent"))


def _child():
    sys.path[:0] = [HERE, os.path.dirname(HERE)]
    import numpy as np

    import workloads as W
    from phd_gb300.izem import IzemGPU
    if sys.argv[1] == "part" and not _green_context(SMS):
        return UNSUPPORTED
    cfg, thd, adi, dxi, st, info, orc = W.case("tgv", 48)
    g = IzemGPU(cfg, thd, adi)
    g.set_grid(*dxi)
    g.upload(**st)
    for _ in range(2):
        g.rk3(g.timestep()[1])
    got = g.download()
    g.close()
    np.savez(sys.argv[2], **{k: got[k] for k in ("v", "T", "cp")})
    return 0


@pytest.mark.gpu
def test_step_on_a_part_of_the_sms(tmp_path):
    import numpy as np
    out = {}
    for which in ("whole", "part"):
        f = str(tmp_path / (which + ".npz"))
        r = subprocess.run([sys.executable, os.path.abspath(__file__), which, f], capture_output=True, text=True, timeout=300)
        if r.returncode == UNSUPPORTED:
            pytest.skip("no green context here: " + r.stdout.strip())
        assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-2000:]
        out[which] = dict(np.load(f))
    for k, want in out["whole"].items():
        np.testing.assert_array_equal(out["part"][k], want)


if __name__ == "__main__":
    sys.exit(_child())
