"""GPU: the table cache holds what a prover goes back and forth between, and
gives way when the library needs the memory."""
import pytest

from oracle import bigref as B

pytestmark = pytest.mark.gpu


def elements(torch, n, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    a = torch.randint(-(1 << 63), (1 << 63) - 1, (n, 4), generator=g, device="cuda", dtype=torch.int64)
    a[:, 3] = torch.randint(0, B.R_MOD >> 192, (n,), generator=g, device="cuda", dtype=torch.int64)
    return a


@pytest.fixture
def builds(zk):
    """tables built on the device so far, as a serving loop reports them"""
    server = zk.Server(hbm_budget=1 << 28)
    yield lambda: server.stats()["table_builds"]
    server.close()


@pytest.mark.parametrize("log_n,log_ext", [(24, 26), (24, 27)])
def test_the_largest_extension_and_the_way_back_build_their_tables_once(zk, oracle, builds, log_n, log_ext):
    torch = pytest.importorskip("torch")
    zk.release_cached()
    torch.cuda.empty_cache()
    n = 1 << log_n
    w, we = oracle.omega(log_n), oracle.omega(log_ext)
    wi, d, g = oracle.inv(w), oracle.inv(oracle.to_mont(n)), oracle.to_mont(7)
    wei, de, gi = oracle.inv(we), oracle.inv(oracle.to_mont(1 << log_ext)), oracle.inv(oracle.to_mont(7))
    vals = elements(torch, n, log_ext)
    ext = torch.empty((1 << log_ext, 4), dtype=torch.int64, device="cuda")
    coeffs = torch.empty_like(vals)
    seen = []
    for _ in range(3):
        zk.lagrange_to_extended_dev(vals, ext, log_n, log_ext, wi, d, g, we)
        zk.extended_to_coeff_dev(ext, coeffs, log_ext, wei, de, gi)
        seen.append(builds())
    torch.cuda.synchronize()
    assert seen[1] == seen[0] and seen[2] == seen[0], seen
    zk.ntt_dev(vals, log_n, wi, post_scale=d)
    assert torch.equal(coeffs, vals)
    del ext, coeffs, vals
    zk.release_cached()
    torch.cuda.empty_cache()


def fill_up_to(torch, left):
    """a tensor that leaves about `left` bytes of the device's memory free"""
    free, _ = torch.cuda.mem_get_info()
    return torch.empty(max(free - left, 0), dtype=torch.uint8, device="cuda")


@pytest.mark.parametrize("what", ["tables", "scratch"])
def test_cached_tables_give_way(zk, oracle, what):
    torch = pytest.importorskip("torch")
    zk.release_cached()
    torch.cuda.empty_cache()
    a = torch.zeros((1 << 26, 4), dtype=torch.int64, device="cuda")
    zk.ntt_dev(a, 26, oracle.omega(26))  # tables of 4.1 GiB, scratch of 2 GiB that stays in the pool
    torch.cuda.synchronize()
    n = 3 << 20  # an MSM with 3.9 GB of scratch
    scalars = torch.ones((n, 4), dtype=torch.int64, device="cuda")
    points = torch.zeros((n, 8), dtype=torch.int64, device="cuda")
    out = torch.full((12,), 1, dtype=torch.int64, device="cuda")
    hog = fill_up_to(torch, 1 << 30)
    if what == "tables":  # of 2 GiB
        zk.ntt_dev(a[:1 << 25], 25, oracle.omega(25))
    else:  # of more than the pool and the free memory have
        zk.msm_dev(scalars, points, out)
    torch.cuda.synchronize()
    assert not a.any().item()
    assert what == "tables" or not out.any().item()
    del hog
    zk.release_cached()
    torch.cuda.empty_cache()
