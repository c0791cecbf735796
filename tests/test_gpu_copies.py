"""Host copies through the page-locked slots: sizes at the edges of the staged
path and of a slot, unaligned host addresses, page-locked arrays, several threads
at once (more than there are staging blocks), and the energies' conversion on the
way (on the device for maps below the staged size, and on the staged path)."""

import ctypes as C
import threading

import numpy as np
import pytest

import parity
import scenes
from ggems_b200 import abi

pytestmark = pytest.mark.gpu

STAGED = 48 << 20  # kStagedCopyBytes
SIZES = [1, 524_289, STAGED - 1, STAGED, STAGED + 1, STAGED + 524_288, 70_000_001]


@pytest.fixture(scope="module", autouse=True)
def staging():
    """A volume that stays, and copies enough for the staging block to be made and kept."""
    from ggems_b200._native import Volume, check, lib
    n = 256 << 20
    src = np.zeros(n, np.uint8)
    v = Volume(abi.GG_MET_UCHAR, (n, 1, 1), (1.0, 1.0, 1.0))
    check(lib.gg_volume_upload(v.handle, C.c_void_p(src.ctypes.data), n))
    yield
    v.close()


def _round_trip(n, seed, offset=0, pinned=False):
    from ggems_b200._native import Volume, check, lib
    rng = np.random.default_rng(seed)
    src = rng.integers(0, 256, n + offset, dtype=np.uint8)[offset:]
    if pinned:
        import torch
        back = torch.empty(n, dtype=torch.uint8, pin_memory=True).numpy()
    else:
        back = np.empty(n + offset, np.uint8)[offset:]
    v = Volume(abi.GG_MET_UCHAR, (n, 1, 1), (1.0, 1.0, 1.0))
    check(lib.gg_volume_upload(v.handle, C.c_void_p(src.ctypes.data), n))
    check(lib.gg_volume_download(v.handle, C.c_void_p(back.ctypes.data), n))
    v.close()
    return np.array_equal(src, back)


@pytest.mark.parametrize("n", SIZES)
def test_round_trip(n):
    assert _round_trip(n, 1)
    assert _round_trip(n, 2, offset=3)


def test_page_locked_and_threads():
    assert _round_trip(STAGED + 5, 3, pinned=True)
    ok = [False] * 4

    def work(k):
        ok[k] = all(_round_trip(STAGED + 777 * k, 10 + k) for _ in range(3))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(ok))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert all(ok)


@pytest.mark.parametrize("n", [16, 200])
def test_energies_are_converted_on_the_way(n):
    """The int64 tally on the device, divided by 2^32, whatever path the copy takes
    (200^3 dosels are 64 MB)."""
    import torch
    from ggems_b200 import _native
    from ggems_b200.distributed import device_tallies
    sc = scenes.water_box_scene(n=n, voxel=128.0 / n)
    src = scenes.XRaySource(monoenergy=scenes.F(60.0) * scenes.KEV, aperture_deg=6.0)
    ctx = _native.Context(0)
    try:
        _, T, _ = parity.run_gpu(ctx, sc, src, 20000)
        q = device_tallies(ctx.handle)[0].cpu().numpy()
        assert q.dtype == np.int64 and q.any()
        want = q.astype(np.float64) / 4294967296.0
        assert np.array_equal(T.edep[0], want)
        # page-locked arrays (200^3: in two pieces of the device's scratch)
        pinned = abi.Tallies([], [n ** 3], alloc=lambda k, t: torch.zeros(
            k, dtype={np.int32: torch.int32, np.float64: torch.float64}[t], pin_memory=True).numpy())
        ctx.read_tallies(pinned)
        assert np.array_equal(pinned.edep[0], want)
        assert np.array_equal(pinned.hit[0], T.hit[0]) and np.array_equal(pinned.edep_squared[0], T.edep_squared[0])
    finally:
        ctx.close()


@pytest.mark.parametrize("last", [False, True])
def test_partly_page_locked_array_is_refused(last):
    """An energy array of which one page only is page-locked: an error before
    anything is written, and the context goes on working."""
    import torch
    from ggems_b200 import _native
    sc = scenes.water_box_scene(n=64, voxel=2.0)
    src = scenes.XRaySource(monoenergy=scenes.F(60.0) * scenes.KEV, aperture_deg=6.0)
    page = 4096
    ctx = _native.Context(0)
    try:
        _, T, _ = parity.run_gpu(ctx, sc, src, 20000)
        raw = np.zeros(64 ** 3 * 8 + 2 * page, np.uint8)
        at = -raw.ctypes.data % page
        edep = raw[at:at + 64 ** 3 * 8].view(np.float64)
        partly = abi.Tallies([], [64 ** 3])
        partly.edep[0] = edep
        partly._ek[0] = abi.ptr(edep, C.c_double)
        locked = edep.ctypes.data + (edep.nbytes - page if last else 0)
        rt = torch.cuda.cudart()
        assert int(rt.cudaHostRegister(locked, page, 0)) == 0
        try:
            with pytest.raises(RuntimeError):
                ctx.read_tallies(partly)
            assert not edep.any()
        finally:
            assert int(rt.cudaHostUnregister(locked)) == 0
        ctx.read_tallies(partly)
        assert np.array_equal(edep, T.edep[0])
    finally:
        ctx.close()


@pytest.mark.parametrize("n", [0, 1, 1000, abi.GG_MAXIMUM_PARTICLES - 1, abi.GG_MAXIMUM_PARTICLES])
def test_random_states_of_some_slots(n):
    """The first n slots of the five arrays go up and come back; the others stay."""
    from ggems_b200 import _native
    S = abi.GG_MAXIMUM_PARTICLES
    ctx = _native.Context(0)
    try:
        first, then = (np.random.default_rng(k).integers(0, 1 << 32, (5, S), dtype=np.uint32) for k in (1, 2))
        ctx.set_random_states(first)
        _native.check(_native.lib.gg_set_random_states(ctx.handle, abi.ptr(then, C.c_uint32), n))
        want = first.copy()
        want[:, :n] = then[:, :n]
        back = np.zeros((5, S), np.uint32)
        ctx.get_random_states(back)
        assert np.array_equal(back, want)
        some = np.zeros((5, S), np.uint32)
        _native.check(_native.lib.gg_get_random_states(ctx.handle, abi.ptr(some, C.c_uint32), n))
        assert np.array_equal(some[:, :n], want[:, :n]) and not some[:, n:].any()
    finally:
        ctx.close()


@pytest.mark.parametrize("mb", [50, 64, 300])
def test_before_and_after_the_block_is_made(mb):
    """In a process of its own: copies of one volume, the first ones by the
    driver and the later ones through a block made meanwhile, and again after
    the last holder has gone."""
    import subprocess
    import sys
    code = """
import ctypes as C, numpy as np
from ggems_b200 import abi
from ggems_b200._native import Volume, check, lib
n = (%d << 20) + 5
for again in range(2):
    v = Volume(abi.GG_MET_UCHAR, (n, 1, 1), (1.0, 1.0, 1.0))
    for k in range(5):
        src = np.random.default_rng(10 * again + k).integers(0, 256, n, dtype=np.uint8)
        check(lib.gg_volume_upload(v.handle, C.c_void_p(src.ctypes.data), n))
        back = np.empty(n, np.uint8) if k %% 2 else np.zeros(n, np.uint8)
        check(lib.gg_volume_download(v.handle, C.c_void_p(back.ctypes.data), n))
        assert np.array_equal(src, back), (again, k)
    v.close()
print("ok")
""" % mb
    out = subprocess.run([sys.executable, "-c", code], cwd=scenes.ROOT, capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and "ok" in out.stdout, out.stderr
