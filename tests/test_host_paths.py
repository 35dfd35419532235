"""Host paths of libkg_b200.so that a GPU test cannot reach -- limits of launches,
refused allocations and launches, a second device -- on the library's own objects
linked with a CUDA runtime that launches nothing (fake_cudart.cpp)."""
import ctypes as C
import os
import shutil
import subprocess
import time

import pytest

from kg_b200 import capi

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("the library's objects cannot be brought up to date here: no nvcc")
    subprocess.run(["make", "-s", "-C", os.path.join(ROOT, "kg_b200", "csrc"), "-j4"], check=True)
    objdir = os.path.join(ROOT, "_build", "kg")
    src = os.path.join(ROOT, "kg_b200", "csrc")
    objs = [os.path.join(objdir, f[:-3] + ".o") for f in sorted(os.listdir(src)) if f.endswith(".cu")]
    out = str(tmp_path_factory.mktemp("fake") / "libkg_fake.so")
    include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    # -Bsymbolic: the runtime calls bind here even when the real runtime is loaded as well
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-I", include,
                    os.path.join(HERE, "fake_cudart.cpp"), *objs, "-o", out,
                    "-Wl,-Bsymbolic,--no-undefined", "-lpthread"], check=True)
    lib = C.CDLL(out)
    for name, restype, argtypes in capi.SIGNATURES:
        f = getattr(lib, name)
        f.restype, f.argtypes = restype, argtypes
    lib.fake_refuse_alloc.argtypes = [C.c_size_t]
    lib.fake_refuse_kernel.argtypes = [C.c_char_p]
    lib.fake_launches.argtypes = [C.c_char_p]
    return lib


class Solve:
    def __init__(self, lib, Nx, Ny, Nz, device=0, metric=capi.KG_KERR_SCHILD):
        self.lib, self.h = lib, C.c_void_p()
        lib.fake_reset()
        p = capi.KgParams(Nx=Nx, Ny=Ny, Nz=Nz, g_pts=2, xmin=1.8, xmax=20.0, tmax=1.0, CFL=0.25, M_bh=1.0, m=0.3,
                          metric=metric, bc_rmax=capi.KG_OUTFLOW, n_det=2, l_max=2, save_=0.1)
        assert lib.kg_create(C.byref(p), device, C.byref(self.h)) == capi.KG_OK

    def __enter__(self):
        return self

    def __exit__(self, *exc):
        self.lib.kg_destroy(self.h)
        self.lib.fake_reset()

    def __call__(self, name, *args):
        """status and error text of an entry point"""
        rc = getattr(self.lib, name)(self.h, *args)
        return rc, self.lib.kg_last_error(self.h).decode()


@pytest.mark.parametrize("pairs", [0, 2])
@pytest.mark.parametrize("Nz", [65534, 65535, 65536, 65537, 70000])
def test_rk4_takes_more_planes_than_a_launch_has_blocks_in_z(fake, Nz, pairs):
    with Solve(fake, 4, 5, Nz) as s:
        assert s("kg_set_rk4_pairs", pairs)[0] == capi.KG_OK
        assert s("kg_rk4", 1) == (capi.KG_OK, "")
        assert s("kg_rk4", 3) == (capi.KG_OK, "")


def test_refused_pole_rows_leave_the_four_stages(fake):
    """no room for the pairs' pole rows: asked for once, outside any capture, and no
    error of a step that the four stage kernels then take"""
    Nx, Ny, Nz = 300, 30, 60
    with Solve(fake, Nx, Ny, Nz) as s:
        assert s("kg_set_rk4_pairs", 2)[0] == capi.KG_OK
        fake.fake_refuse_alloc(10 * (Nz + 1) * ((Nx + 5 + 7) // 8 * 8) * 16)
        for n in (6, 6, 1, 3):
            assert s("kg_rk4", n) == (capi.KG_OK, "")
        assert fake.fake_refused() == 2  # dalloc tries again behind a trim of the pool
        assert fake.fake_capture_allocs() == 0
        assert fake.fake_launches(b"rk4_pair") == 0
        assert fake.fake_launches(b"tma_stage") > 0


@pytest.mark.parametrize("metric", [capi.KG_KERR_SCHILD, capi.KG_SCHW_EF])
def test_every_kernel_launches_on_a_second_device(fake, metric):
    """what a launch needs is set on the device that launches, not once a process"""
    seen = []
    for device in (0, 1):
        with Solve(fake, 60, 12, 20, device=device, metric=metric) as s:
            for name in ("kg_pirk2", "kg_pirk3", "kg_rk3", "kg_rk4"):
                assert s(name, 1) == (capi.KG_OK, "")
            for rows in (4, 8):
                for precision in (0, 1):
                    for pairs in (0, 2):
                        s("kg_set_tile_rows", rows), s("kg_set_precision", precision), s("kg_set_rk4_pairs", pairs)
                        assert s("kg_rk4", 2) == (capi.KG_OK, "")
                    b = C.c_void_p()
                    assert fake.kg_batch_create(device, C.byref(b)) == capi.KG_OK
                    assert fake.kg_batch_set_precision(b, precision) == capi.KG_OK
                    assert fake.kg_batch_set_tile_rows(b, rows) == capi.KG_OK
                    assert fake.kg_batch_add(b, s.h) == capi.KG_OK
                    assert fake.kg_batch_rk4(b, 2) == capi.KG_OK, fake.kg_batch_last_error(b)
                    assert fake.kg_batch_destroy(b) == capi.KG_OK
            alm = (C.c_double * (2 * 3 * 5 * 60))()
            assert s("kg_project_all_shells", 2, 1, alm) == (capi.KG_OK, "")
            if metric == capi.KG_KERR_SCHILD:
                assert s("kg_set_precision", 0)[0] == s("kg_set_scheme", 1, 0.02)[0] == capi.KG_OK
                assert s("kg_rk4", 2) == (capi.KG_OK, "")
            seen.append([fake.fake_launches(k)
                         for k in (b"tma_stage", b"tma_batch", b"mx_stage", b"mx_batch", b"rk4_pair", b"pirk_s1_fused",
                                   b"cfg_march", b"ylm_gemm", b"2kg12march_kernel")])
    assert seen[0] == seen[1] and all(seen[0][:6]) and not seen[0][-1]


REFUSED = [("tma_stage_kernel", "kg_pirk2", "2kg12march_kernel"), ("tma_stage_kernel", "kg_pirk3", "2kg12march_kernel"),
           ("tma_stage_kernel", "kg_rk3", "2kg12march_kernel"), ("tma_stage_kernel", "kg_rk4", "2kg12march_kernel"),
           ("pirk_s1_fused", "kg_pirk2", "tma_stage_kernel"), ("pirk_s1_fused", "kg_pirk3", "tma_stage_kernel"),
           ("cfg_march_kernel", "configured", "cfg_stage_kernel"),
           ("rk4_pair_kernelILi0", "paired", "tma_stage_kernel"), ("rk4_pair_kernelILi1", "paired", "tma_stage_kernel")]


@pytest.mark.parametrize("kernel,call,instead", REFUSED)
@pytest.mark.parametrize("later", [False, True])
def test_refused_launch_takes_the_other_form(fake, kernel, call, instead, later):
    """a launch that the device refuses -- at once, or behind steps that it took -- is
    no error of a step that another form takes, nor of the calls after it"""
    with Solve(fake, 40, 12, 20) as s:
        name = call if call.startswith("kg_") else "kg_rk4"
        assert s("kg_set_rk4_pairs", 2 if call == "paired" else 0)[0] == capi.KG_OK
        if call == "configured":
            assert s("kg_set_scheme", 1, 0.02)[0] == capi.KG_OK
        assert s(name, 3 if later else 0)[0] == capi.KG_OK
        sc = (C.c_double * 9)()
        assert s("kg_get_scalars", sc)[0] == capi.KG_OK
        t, dt = sc[4], sc[3]
        fake.fake_refuse_kernel(kernel.encode())
        before = fake.fake_launches(instead.encode())
        assert s("kg_set_graphs", 0)[0] == capi.KG_OK
        for n in (1, 4, 3):
            assert s(name, n) == (capi.KG_OK, "")
            for _ in range(n):
                t = t + dt
        assert fake.fake_launches(instead.encode()) > before
        assert s("kg_get_scalars", sc)[0] == capi.KG_OK and sc[4] == t
        fake.fake_refuse_kernel(None)
        assert s(name, 2) == (capi.KG_OK, "")
        assert fake.fake_last_error() == 0


@pytest.mark.parametrize("kernel", ["mx_stage_kernelILi9", "mx_stage_kernelILi11"])
def test_refused_mixed_stage_does_not_fail_the_next_call(fake, kernel):
    with Solve(fake, 40, 12, 20) as s:
        assert s("kg_set_precision", 1)[0] == capi.KG_OK
        fake.fake_refuse_kernel(kernel.encode())
        assert s("kg_rk4", 1)[0] == capi.KG_ECUDA
        assert s("kg_pirk2", 1)[0] == capi.KG_OK


@pytest.mark.parametrize("method", ["kg_pirk2", "kg_pirk3", "kg_rk3", "kg_rk4"])
def test_host_time_of_a_step_does_not_grow_with_the_planes(fake, method):
    """the chunk rule runs at every launch: a step of a grid with many planes is
    enqueued in the microseconds of its launches (about 50), not in a search over all
    numbers of chunks (5 to 14 ms here)"""
    with Solve(fake, 4, 5, 200000) as s:
        best = 1.0
        for _ in range(6):
            t0 = time.perf_counter()
            assert s(method, 1)[0] == capi.KG_OK
            best = min(best, time.perf_counter() - t0)
        assert best < 1e-3


def test_chunk_rules_equal_the_search_over_all_numbers_of_chunks(tmp_path):
    src, so = tmp_path / "c.cpp", str(tmp_path / "c.so")
    src.write_text('#include "kg_chunk.h"\n'
                   'extern "C" int phi(int p, int t, int s, int l) { return kg::phi_chunk(p, t, s, l); }\n'
                   'extern "C" int pair(int p, int t) { return kg::pair_chunk(p, t); }\n')
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-I", os.path.join(ROOT, "kg_b200", "csrc"),
                    str(src), "-o", so], check=True)
    lib = C.CDLL(so)

    def search(planes, longest, cost):
        tried = [-(-planes // n) for n in range(-(-planes // longest), planes + 1)]
        return min(((cost(c, -(-planes // c)), i, c) for i, c in enumerate(tried)))[2]

    for planes in [*range(1, 70), 128, 129, 256, 257, 333, 1025]:
        for tiles in (1, 2, 3, 7, 12, 40, 90, 111, 148, 296, 297, 1000, 4321):
            for slots, longest in ((296, 32), (444, 32), (296, 64)):
                want = search(planes, longest, lambda c, m: max(tiles * m / slots + 0.25, 1.0) * (c + 1))
                assert lib.phi(planes, tiles, slots, longest) == want
            want = search(planes, 24, lambda c, m: ((tiles * m + 147) // 148 + 0.5) * (c + 3))
            assert lib.pair(planes, tiles) == want


@pytest.mark.parametrize("grid,two,one", [((64, 17, 33), 0, 0), ((64, 65, 129), 0, 0), ((512, 33, 65), 4, 0),
                                          ((1024, 65, 129), 4, 2)])
def test_rk4_steps_by_pairs_where_they_pay(fake, grid, two, one):
    """pair kernels of two steps in a call and of one, which needs a copy of u as well"""
    with Solve(fake, *grid) as s:
        assert s("kg_set_graphs", 0)[0] == capi.KG_OK
        assert s("kg_rk4", 1)[0] == capi.KG_OK  # fills the seam planes
        for n, want in ((2, two), (1, one), (3, two + one), (1, one)):
            before = fake.fake_launches(b"rk4_pair")
            assert s("kg_rk4", n)[0] == capi.KG_OK
            assert fake.fake_launches(b"rk4_pair") - before == want


@pytest.mark.parametrize("n", range(2, 9))
def test_rk4_kernels_run_once_ahead_of_their_capture(fake, n):
    with Solve(fake, 512, 33, 65) as s:
        before = [fake.fake_launches(k) for k in (b"rk4_pair", b"tma_stage")]
        assert s("kg_rk4", n) == (capi.KG_OK, "")
        steps = [fake.fake_launches(k) - b for k, b in zip((b"rk4_pair", b"tma_stage"), before)]
        # one step that fills the seam planes, two direct ones, two in the capture, an odd last one by stages
        left = n - 1 if n < 5 else 4 + (n - 3) % 2
        assert steps == [4 * (left // 2), 4 * (1 + left % 2)]


@pytest.mark.parametrize("method", ["kg_rk3", "kg_rk4"])
@pytest.mark.parametrize("grid", [(40, 9, 17), (128, 33, 65), (1024, 65, 129)])
def test_stages_store_their_ghost_values_on_a_filled_state(fake, method, grid):
    with Solve(fake, *grid) as s:
        assert s("kg_set_rk4_pairs", 0)[0] == s("kg_set_graphs", 0)[0] == capi.KG_OK
        assert s(method, 1)[0] == capi.KG_OK
        fills = fake.fake_launches(b"ghost_kernel")
        assert fills > 0
        assert s(method, 3)[0] == capi.KG_OK
        assert fake.fake_launches(b"ghost_kernel") == fills


@pytest.mark.parametrize("grid,precision,want", [((64, 17, 33), 0, 1360), ((1024, 65, 129), 0, 560),
                                                 ((1024, 65, 129), 1, 880)])
def test_step_bytes_follow_the_kernels(fake, grid, precision, want):
    from kg_b200.profile_cases import step_bytes
    with Solve(fake, *grid) as s:
        b = C.c_void_p()
        assert fake.kg_batch_create(0, C.byref(b)) == fake.kg_batch_set_precision(b, precision) == capi.KG_OK
        assert fake.kg_batch_set_dispatch(b, 1, -1) == fake.kg_batch_add(b, s.h) == capi.KG_OK
        assert fake.kg_batch_rk4(b, 1) == capi.KG_OK
        assert step_bytes(fake, [s.h], lambda: fake.kg_batch_rk4(b, 2), 2) == [want]
        fake.kg_batch_destroy(b)


def test_every_stage_kernel_has_its_bytes(fake):
    from kg_b200.profile_cases import STAGE_BYTES
    names = [fake.kg_profile_kind_name(i).decode() for i in range(fake.kg_profile_kinds())]
    assert {n for n in names if n.startswith(("stage_", "mixed_"))} == set(STAGE_BYTES)
