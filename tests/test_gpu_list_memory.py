"""The memory of neighbour lists (GPU): a list can be exported to another
process, as any allocation of its own; a freed list's block serves the next list
of about its length, and what is kept beyond 2 GB goes back to the driver, as does
what the library's pool holds unused above 6 GB."""
import ctypes as C
import threading

import numpy as np
import pytest

from helpers import random_box

pytestmark = pytest.mark.gpu

GB = 1 << 30


def gas(torch, n, neighbours, seed):
    """(n, 3) float32 positions on the GPU, sites of a sparse grid, and the box side at cutoff 1."""
    side = float(np.float32((n * 4.0 / 3.0 * np.pi / neighbours) ** (1.0 / 3.0)))
    m = int(np.ceil((n / 0.8) ** (1.0 / 3.0)))
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    site = torch.randperm(m ** 3, generator=g, device="cuda")[:n]
    cell = torch.stack([site % m, site // m % m, site // (m * m)], 1).float()
    x = (cell + torch.rand((n, 3), generator=g, device="cuda") * 0.9) * (side / m)
    x[x >= side] = 0.0
    return x.contiguous(), side


def free_bytes(torch):
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.cuda.mem_get_info()[0]


def test_export_to_another_process(built_lib):
    """cudaIpcGetMemHandle takes the list's address."""
    torch = pytest.importorskip("torch")
    import irregular_gb300 as irr
    torch.zeros(1, device="cuda")
    pos, side = random_box(5000, 0.9, 1)
    lst = irr.neighbor_build(pos, float(side), 6.25)
    cudart = irr._cudart()
    handle = (C.c_char * 64)()
    assert cudart.cudaIpcGetMemHandle(handle, C.c_void_p(lst.ptr)) == 0
    lst.close()


def test_next_list(built_lib, oracle_lib):
    """Blocks taken again hold the next list, whatever was in them; lists of
    several lengths live at once are apart."""
    import irregular_gb300 as irr
    want = {}
    for k, n in enumerate([4000, 4100, 900, 30000, 3900, 29000]):
        pos, side = random_box(n, 0.9, k)
        want[n] = (pos, float(side), oracle_lib.neighbor_half_list(pos, float(side), np.float32(6.25)))
    rng = np.random.default_rng(3)
    live = []
    for _ in range(200):
        n = int(rng.choice(list(want)))
        pos, side, ref = want[n]
        live.append((irr.neighbor_build(pos, side, 6.25), ref))
        if len(live) > 4:
            got, ref = live.pop(int(rng.integers(len(live))))
            assert np.array_equal(got.to_host(), ref)
            got.close()
    spans = sorted((x.ptr, x.ptr + 8 * x.count) for x, _ in live)
    assert all(a[1] <= b[0] for a, b in zip(spans, spans[1:]))
    for got, ref in live:
        assert np.array_equal(got.to_host(), ref)
        got.close()


@pytest.mark.parametrize("n", [50, 2916, 20_000, 300_000])
def test_same_block_again(built_lib, n):
    """A list made and freed again and again keeps its block, whatever its length."""
    import irregular_gb300 as irr
    pos, side = random_box(n, 0.9, n)
    seen = set()
    for _ in range(6):
        lst = irr.neighbor_build(pos, float(side), 6.25)
        seen.add(lst.ptr)
        lst.close()
    assert len(seen) == 1


def test_several_threads(built_lib, oracle_lib):
    """Lists made and freed by six threads at once, from the same kept blocks."""
    import irregular_gb300 as irr
    want = []
    for k, n in enumerate([3000, 3050, 12_000, 700]):
        pos, side = random_box(n, 0.9, k)
        want.append((pos, float(side), oracle_lib.neighbor_half_list(pos, float(side), np.float32(6.25))))
    failed = []

    def work(t):
        rng = np.random.default_rng(t)
        try:
            held = []
            for _ in range(80):
                pos, side, ref = want[int(rng.integers(len(want)))]
                held.append((irr.neighbor_build(pos, side, 6.25), ref))
                if len(held) > 2:
                    got, ref = held.pop(int(rng.integers(len(held))))
                    assert np.array_equal(got.to_host(), ref)
                    got.close()
            for got, ref in held:
                assert np.array_equal(got.to_host(), ref)
                got.close()
        except BaseException as e:  # noqa: BLE001 -- told to the test's own thread
            failed.append(repr(e))

    threads = [threading.Thread(target=work, args=(t,)) for t in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed


def test_freed_twice(built_lib, oracle_lib):
    """The second free is refused, and the block is not given out twice."""
    import irregular_gb300 as irr
    pos, side = random_box(4000, 0.9, 2)
    want = oracle_lib.neighbor_half_list(pos, float(side), np.float32(6.25))
    first = irr.neighbor_build(pos, float(side), 6.25)
    ptr, free = C.c_void_p(first.ptr), irr.load().irr_device_free
    assert free(0, ptr) == irr.IRR_OK
    assert free(0, ptr) == irr.IRR_ERR_CUDA
    first.ptr = 0
    lists = [irr.neighbor_build(pos, float(side), 6.25) for _ in range(3)]
    assert len({x.ptr for x in lists}) == 3
    for x in lists:
        assert np.array_equal(x.to_host(), want)
        x.close()


def test_freed_lists_go_back(built_lib):
    torch = pytest.importorskip("torch")
    import irregular_gb300 as irr
    pos, side = gas(torch, 5_000_000, 64, 2)
    irr.neighbor_build(pos, side, 1.0).close()  # the pool's temporaries, and one list's block
    before = free_bytes(torch)
    lists = [irr.neighbor_build(pos, side, 1.0) for _ in range(4)]
    size = 8 * lists[0].count
    assert size > GB
    assert before - free_bytes(torch) > 2.9 * size
    for x in lists:
        x.close()
    assert before - free_bytes(torch) < 2 * GB + 0.1 * size


def test_unused_pool_memory_goes_back(built_lib):
    """A list whose slots alone take more than the pool keeps."""
    torch = pytest.importorskip("torch")
    import irregular_gb300 as irr
    pos, side = gas(torch, 24_000_000, 64, 4)
    before = free_bytes(torch)
    irr.neighbor_build(pos, side, 1.0).close()
    assert before - free_bytes(torch) < 8.5 * GB
