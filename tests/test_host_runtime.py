"""The library's host code on a CUDA runtime without a GPU (fake_cudart.cpp):
what it hands to the runtime on first calls and streams.

Each scenario runs in a process of its own, in which the fake takes
libcudart's place before the library loads."""
import ctypes
import json
import os
import subprocess
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    from hilbert_b200 import build
    build.build()
    d = tmp_path_factory.mktemp("fake")
    (d / "version").write_text("libcudart.so.12 { global: cuda*; __cuda*; fake_*; local: *; };\n")
    cuda = os.path.dirname(os.path.dirname(build.nvcc_path()))
    so = str(d / "libcudart.so.12")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", os.path.join(cuda, "include"),
                           os.path.join(HERE, "fake_cudart.cpp"), "-o", so, "-Wl,-soname,libcudart.so.12",
                           f"-Wl,--version-script={d / 'version'}"])

    def run(scenario, *args):
        out = subprocess.run([sys.executable, os.path.abspath(__file__), so, scenario, *map(str, args)],
                             capture_output=True, text=True, timeout=600, cwd=ROOT)
        assert out.returncode == 0, out.stderr[-4000:]
        return json.loads(out.stdout.strip().splitlines()[-1])
    return run


@pytest.mark.parametrize("call", ["Au", "project", "warm", "mode1", "solve", "profiled", "continued", "bpsdp",
                                  "pack"])
def test_uploads_are_waited_for(fake, call):
    """A pageable cudaMemcpy or a cudaMemset may return before the device holds
    its result, and nothing orders the legacy stream they run on with a
    non-blocking one: every table and fill of a problem's first call is waited
    for before work on another stream can read it."""
    out = fake("uploads", call)
    assert out["faults"] == [], out["faults"][:5]
    assert out["launches"] > 0


def test_another_set_of_blocks_uses_no_freed_memory(fake):
    """A host solver may give other block dimensions on its next call: the plan
    is given back and built again, its grown cluster lists included."""
    out = fake("rebuilt")
    assert out["clusters"] >= 2 and out["faults"] == []
    assert out["left"] == 0   # destroyed: nothing stays allocated


@pytest.mark.parametrize("call", ["Au", "project", "warm", "solve", "bpsdp", "pack"])
def test_a_call_after_a_failed_allocation_starts_again(fake, call):
    """Whichever allocation of a first call fails, the call returns an error, and
    the next one makes what is missing: the launches of an undisturbed call, none
    with a null pointer in the place of a table."""
    out = fake("retried", call)
    assert out["tried"] > 10
    assert out["wrong"] == []


@pytest.mark.parametrize("second", ["project", "warm", "solve"])
def test_a_new_stream_with_an_old_handle_waits(fake, second):
    """The work arrays' next user waits for the last one unless it is on the same
    stream, which a handle alone does not tell: that of a destroyed stream is
    given out again while its work may still run."""
    out = fake("reused", second)
    assert out["same_handle"]
    assert out["waits"] == 1
    assert out["waits_on_the_same_stream"] == 0


def test_stand_alone_projections_are_profiled(fake):
    """Profiling level 2 times a stand-alone projection's launches beside the
    solver's (collected by the next solve), but not inside a capture."""
    out = fake("profiled_projection")
    gemm, acceptance = out["project"][0] - out["none"][0], out["project"][1] - out["none"][1]
    assert gemm == out["launched"] and acceptance == 1
    assert out["captured"] == out["none"]


# ---------------------------------------------------------------- scenarios
class Host:
    """The library on the fake runtime; device vectors are numpy arrays."""

    def __init__(self, so):
        import numpy as np
        self.np = np
        self.rt = ctypes.CDLL(so, mode=ctypes.RTLD_GLOBAL)
        self.rt.fake_events.restype = ctypes.c_char_p
        self.rt.fake_fail_at.argtypes = [ctypes.c_long]
        for f in ("fake_allocations", "fake_faults", "fake_live"):
            getattr(self.rt, f).restype = ctypes.c_long
        sys.path.insert(0, ROOT)
        import hilbert_b200 as hb
        from hilbert_b200 import _capi
        assert "torch" not in sys.modules   # its libraries want the real runtime
        self.hb, self.capi = hb, _capi
        self.lib = _capi.load()

    def stream(self):
        s = ctypes.c_void_p()
        self.rt.cudaStreamCreateWithFlags(ctypes.byref(s), 1)
        return s

    def events(self):
        return self.rt.fake_events().decode().splitlines()

    def clear(self):
        self.rt.fake_clear()

    def problem(self, n=3, pos="DQG", doci=False):
        return (self.hb.DOCIProblem if doci else self.hb.V2RDMProblem)(n, 2, 2 if doci else 1, pos)

    def call(self, what, p, stream):
        """the entry point's status"""
        np, lib = self.np, self.lib
        vec = lambda k: np.zeros(k).ctypes.data_as(ctypes.c_void_p)   # noqa: E731
        keep = [np.zeros(max(p.n_primal, p.n_dual)) for _ in range(3)]
        a, b, c = (v.ctypes.data for v in keep)
        if what == "Au":
            return max(lib.v2b_problem_Au(p._h, a, b, stream), lib.v2b_problem_ATu(p._h, a, b, stream))
        if what == "project":
            return lib.v2b_problem_project(p._h, a, 1.0, b, c, stream)
        if what == "mode1":
            lib.v2b_problem_set_projection_mode(p._h, 1)
            return lib.v2b_problem_project(p._h, a, 1.0, b, c, stream)
        if what == "warm":
            return (lib.v2b_problem_project_warm(p._h, a, 1.0, b, c, stream) or
                    lib.v2b_problem_project_warm(p._h, a, 1.0, b, c, stream))
        if what == "pack":
            g = p.n * (p.n + 1) // 2 if hasattr(p, "n") else 6
            out = np.zeros(g * (g + 1) // 2 + g)
            return lib.v2b_problem_pack_spatial_density(p._h, a, out.ctypes.data, out.ctypes.data, stream)
        if what == "profiled":
            rc = lib.v2b_problem_set_profiling(p._h, 2)
            return rc or self.call("solve", p, stream)
        if what == "continued":
            rc = self.call("solve", p, stream)
            return rc or lib.v2b_problem_continue(p._h) or self.call("solve", p, stream)
        assert what == "solve"
        o = self.capi.SDPOptions(1e-6, 1e-6, 1e-9, 100, 4)
        oi, ii, e = ctypes.c_long(), ctypes.c_long(), ctypes.c_double()
        return lib.v2b_problem_solve(p._h, self.dp(keep[0]), self.dp(keep[1]), self.dp(keep[2]), ctypes.byref(o), 2,
                                     self.capi.SDP_MONITOR(), 0, None, ctypes.byref(oi), ctypes.byref(ii),
                                     ctypes.byref(e))

    @staticmethod
    def dp(v):
        return v.ctypes.data_as(ctypes.POINTER(ctypes.c_double))

    def bpsdp(self, dims):
        """a host solver whose maps are the identity: its handle and a solve"""
        np, lib, capi = self.np, self.lib, self.capi
        n = sum(d * d for d in dims)
        h = ctypes.c_void_p()
        o = capi.SDPOptions(1e-6, 1e-6, 1e-9, 3, 4)
        capi.check(lib.v2b_bpsdp_create(n, n, ctypes.byref(o), ctypes.byref(h)))

        def copy(out, v, _):
            ctypes.memmove(out, v, 8 * n)
        cb = capi.SDP_CALLBACK(copy)
        ones = np.ones(n)

        def solve(dims):
            x = np.zeros(n)
            d = (ctypes.c_int * len(dims))(*dims)
            return lib.v2b_bpsdp_solve(h, self.dp(x), self.dp(ones), self.dp(ones), d, len(dims), 2, cb, cb,
                                       capi.SDP_MONITOR(), 0, None)
        return h, solve


def uploads(host, call):
    if call == "bpsdp":
        h, solve = host.bpsdp([4, 30, 200])
        rc = solve([4, 30, 200])
        host.lib.v2b_bpsdp_destroy(h)
    else:
        rc = 0
        for p in (host.problem(), host.problem(5), host.problem(4, doci=True)):
            rc = max(rc, host.call(call, p, host.stream()))
            p.close()
    assert rc in (0, 1), (rc, host.lib.v2b_last_error())
    ev = host.events()
    return {"faults": [e for e in ev if e.startswith("FAULT")], "launches": sum(e.startswith("launch") for e in ev)}


def retried(host, call):
    host.rt.fake_refine_script(1)

    def attempt(k):
        """a fresh object whose first call fails at allocation k: the status of
        that call and of the next, and the next one's launches"""
        if call == "bpsdp":
            h, solve = host.bpsdp([4, 30, 200])
            first = lambda: solve([4, 30, 200])                                # noqa: E731
            done = lambda: host.lib.v2b_bpsdp_destroy(h)                       # noqa: E731
        else:
            p, s = host.problem(6 if call == "project" else 4, doci=call == "pack"), host.stream()
            first = lambda: host.call(call, p, s)                              # noqa: E731
            done = lambda: (p.close(), host.rt.cudaStreamDestroy(s))           # noqa: E731
        host.clear()
        host.rt.fake_fail_at(k)
        rc = [first()]
        count = host.rt.fake_allocations()
        host.rt.fake_fail_at(-1)
        faults = host.rt.fake_faults()
        host.clear()
        rc.append(first())
        ev = host.events()
        done()
        ev += [e for e in host.events() if e.startswith("FAULT")]
        return rc, count, faults, {e for e in ev if e.startswith("launch") or e.startswith("FAULT")}, host.rt.fake_live()

    _, count, _, again, left = attempt(-1)
    # what a first call launches (its autotuner included) and a second one
    host_first = set()
    if call != "bpsdp":
        p, s = host.problem(6 if call == "project" else 4, doci=call == "pack"), host.stream()
        host.clear()
        host.call(call, p, s)
        host_first = {e for e in host.events() if e.startswith("launch")}
        p.close()
        host.rt.cudaStreamDestroy(s)
    else:
        h, solve = host.bpsdp([4, 30, 200])
        host.clear()
        solve([4, 30, 200])
        host_first = {e for e in host.events() if e.startswith("launch")}
        host.lib.v2b_bpsdp_destroy(h)
    known = again | host_first
    wrong = [] if left == 0 else [f"{left} allocations left"]
    for k in range(count):
        rc, _, faults, seen, left = attempt(k)
        if rc[0] != host.capi.V2B_CUDA_ERROR or rc[1] > 1 or faults or not seen <= known or left:
            wrong.append([k, rc, faults, sorted(seen - known)[:3], left])
    return {"tried": count, "wrong": wrong[:5]}


def reused(host, second):
    p, s = host.problem(4), host.stream()
    assert host.call("project", p, s) == 0
    host.clear()
    assert host.call("project", p, s) == 0
    same = host.events().count("wait")
    host.rt.cudaStreamDestroy(s)
    t = host.stream()
    host.clear()
    lib, v = host.lib, host.np.zeros(p.n_primal)
    if second == "warm":   # one call
        rc = lib.v2b_problem_project_warm(p._h, v.ctypes.data, 1.0, v.ctypes.data, v.ctypes.data, t)
    else:
        rc = host.call(second, p, t)
    assert rc <= 1
    return {"same_handle": s.value == t.value, "waits": host.events().count("wait"), "waits_on_the_same_stream": same}


def profiled_projection(host):
    out = {}
    for what in ("none", "project", "captured"):
        p, s = host.problem(6), host.stream()
        assert host.lib.v2b_problem_set_profiling(p._h, 2) == 0
        assert host.call("project", p, s) == 0        # builds the plan and its lists
        assert host.lib.v2b_problem_set_profiling(p._h, 2) == 0
        host.clear()
        host.rt.fake_capture(s, what == "captured")
        if what != "none":
            assert host.call("project", p, s) == 0
        host.rt.fake_capture(s, False)
        if what == "project":   # the small blocks' kernel and the tiles
            out["launched"] = sum("gemm_tiles" in e or "sign_small" in e for e in host.events())
        assert host.call("solve", p, s) <= 1
        ms, n = (ctypes.c_double * 5)(), (ctypes.c_long * 5)()
        assert host.lib.v2b_problem_projection_profile(p._h, ms, n, 5) == 0
        out[what] = list(n)
        p.close()
    return out


def rebuilt(host):
    host.rt.fake_refine_script(1)   # warm blocks form a cluster: its lists live in grown memory
    h, solve = host.bpsdp([30, 40])
    rc = [solve(d) for d in ([30, 40], [40, 30], [30, 40])]
    assert max(rc) <= 1, (rc, host.lib.v2b_last_error())
    host.lib.v2b_bpsdp_destroy(h)
    ev = host.events()
    return {"faults": [e for e in ev if e.startswith("FAULT")], "left": host.rt.fake_live(),
            "clusters": sum("cluster_rows_kernel" in e for e in ev)}


if __name__ == "__main__":
    print(json.dumps(globals()[sys.argv[2]](Host(sys.argv[1]), *sys.argv[3:])))
