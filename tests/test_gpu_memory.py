"""Device memory that a context keeps: the queues of large wavefronts against the free memory, and the bound on what
the device's pool keeps unused (GPU)."""
import pytest

from mobileraytracer_b200 import Context, Scene, capi, scenes

pytestmark = pytest.mark.gpu
GB = 1 << 30


@pytest.fixture
def free_memory():
    """free_memory(bytes): the device's memory filled but for so many; the free bytes then."""
    torch = pytest.importorskip("torch")
    fill = []

    def leave(n):
        torch.cuda.empty_cache()
        have = torch.cuda.mem_get_info(0)[0]
        if have < n:
            pytest.skip("too little free device memory")
        fill.append(torch.empty(have - n, dtype=torch.uint8, device="cuda"))
        return torch.cuda.mem_get_info(0)[0]

    yield leave
    fill.clear()
    torch.cuda.empty_cache()


def _render(ctx, spl, size=2048):
    torch = pytest.importorskip("torch")
    sc = scenes.cornell_box()
    g = Scene(ctx, sc).build()
    opts = capi.render_opts(shader=capi.MRT_SHADER_PATHTRACER, width=size, height=size, spp=1, spl=spl, depth_min=2, depth_max=6)
    bm = torch.zeros(size * size, dtype=torch.int32, device="cuda")
    g.render(sc.camera, opts, bitmap=bm)
    g.close()


# The queues of 2^22 paths at depth 6 are 7.3 GB, 9.1 GB as they are allocated: of 64 GB more than an eighth
# (then 2^21 paths), of 90 GB less
@pytest.mark.parametrize("free,most", [(64, 8), (90, 11.25)])
def test_queues_take_an_eighth_of_the_free_memory(free_memory, free, most):
    torch = pytest.importorskip("torch")
    before = free_memory(free * 10**9)
    c = Context(0)
    _render(c, 1)
    taken = before - torch.cuda.mem_get_info(0)[0]
    c.close()
    slack = 0.2e9   # the context, the scene, the pixels
    assert 4e9 < taken < most * 10**9 + slack
    assert (taken > 8.5e9) == (free == 90)


def test_a_queue_that_has_to_grow_counts(free_memory):
    """2^22 paths with one light sample, then with 32, whose shadow queue alone is 10.7 GB (13.4 as allocated):
    more than an eighth of 90 GB with the others, so the second frame runs 2^21 paths at a time."""
    torch = pytest.importorskip("torch")
    before = free_memory(90 * 10**9)
    c = Context(0)
    _render(c, 1)
    _render(c, 32)
    taken = before - torch.cuda.mem_get_info(0)[0]
    c.close()
    assert taken < 17e9
