"""Host side of a solve on the fake runtime of fake_cudart.cpp, in a process of
its own (the fake takes the place of libcudart.so, so nothing here imports
torch): ``python host_dispatch.py <fake library> <json list of steps>`` prints
one JSON list with each step's status and launches."""

import ctypes
import json
import os
import sys
import types

import numpy as np

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def main(fake_path, steps):
    fake = ctypes.CDLL(fake_path, mode=ctypes.RTLD_GLOBAL)  # before the library: takes libcudart's place
    fake.fake_log.restype = ctypes.c_char_p
    sys.path.insert(0, ROOT)
    pkg = types.ModuleType("easyfea_gb300")  # without the package's imports of torch
    pkg.__path__ = [os.path.join(ROOT, "easyfea_gb300")]
    sys.modules["easyfea_gb300"] = pkg
    from easyfea_gb300 import _lib

    L = _lib.load()
    out = []
    for s in steps:
        fake.fake_device(s.get("device", 0), s.get("sms", 152), s.get("coop_limit", s.get("sms", 152)))
        fake.fake_timed_out(s.get("timed_out", 0))
        L.gfea_tune_mode(s.get("tune_mode", 1))
        for k in ("GFEA_STAGE_MIN_BYTES", "GFEA_RESIDENT_CTAS"):
            os.environ.pop(k, None)
        os.environ.update(s.get("env", {}))
        D, Nn, deg = s["D"], s["nodes"], s["degree"]
        prec = _lib.F32 if s["precision"] == "mixed" else _lib.F64
        # kernels do not run: only pointers, counts and sizes matter
        a = {"ptr": np.zeros(Nn + 1, np.int32), "known": np.zeros(Nn * D, np.uint8), "coord": np.zeros(3 * Nn),
             "v": np.zeros(8), "b": np.zeros(Nn * D), "x": np.zeros(Nn * D)}
        p = {k: v.ctypes.data for k, v in a.items()}
        sysd = _lib.System(_lib.ABI_VERSION, D, Nn, Nn * deg, p["ptr"], p["ptr"], p["v"], p["v"], p["known"], 0, 0,
                           p["coord"])
        opts = _lib.PcgOpts(_lib.ABI_VERSION, prec, 100, s.get("check_every", 0), 1e-10, 0.0, 10, s.get("lanes", 0),
                            s.get("coarse", -1), 0)
        ws = ctypes.c_size_t()
        if s.get("work_without_tiles"):  # the size that a smaller threshold's operator would need
            os.environ["GFEA_STAGE_MIN_BYTES"] = str(1 << 60)
        assert L.gfea_pcg_workspace_size(ctypes.byref(sysd), ctypes.byref(opts), ctypes.byref(ws)) == 0
        os.environ.pop("GFEA_STAGE_MIN_BYTES", None)
        os.environ.update(s.get("env", {}))
        work = np.zeros(ws.value + 256, np.uint8)
        base = (work.ctypes.data + 255) & ~255
        res = _lib.PcgResult()
        fake.fake_clear()
        st = L.gfea_pcg_solve(ctypes.byref(sysd), p["b"], p["x"], ctypes.byref(opts), base, ws.value,
                              ctypes.byref(res), 0)
        out.append({"status": st, "result": res.status, "launches": fake.fake_log().decode().splitlines()})
    print(json.dumps(out))


if __name__ == "__main__":
    main(sys.argv[1], json.loads(sys.argv[2]))
