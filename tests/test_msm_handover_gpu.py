"""GPU: the last step of zkgpu_msm_dev, which the stream's last kernel hands to
a thread of the library and otherwise does itself (msm_combine.cu).  Every
case runs in a process of its own, since ZKGPU_MSM_HOST_WAIT_US is read once;
results are compared with the oracle here."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PRELUDE = """
import sys, threading, time
import numpy as np, torch
import zk_gpu_b200 as zk
data = np.load(sys.argv[1])
ds, db = (torch.from_numpy(data[k].view(np.int64)).cuda() for k in ("s", "b"))
save = lambda x: np.save(sys.argv[2], x.cpu().numpy().view(np.uint64))
"""


def run_child(tmp_path, code, s, pts, **env):
    inp, out = str(tmp_path / "in.npz"), str(tmp_path / "out.npy")
    np.savez(inp, s=s, b=pts)
    subprocess.run([sys.executable, "-c", PRELUDE + code, inp, out], cwd=ROOT, env=dict(os.environ, **env),
                   check=True, timeout=300)
    return np.load(out)


@pytest.mark.parametrize("wait_us", ["0", "3000"])
def test_result_pointer_aligned_to_its_words_only(oracle, tmp_path, wait_us):
    """d_out_xyz is an array of 64-bit words and may start at any of them,
    whoever does the last step; the sum over no points too."""
    n = 100
    s, pts = oracle.rand_fr(n, 901), oracle.rand_bases(n, 902)
    got = run_child(tmp_path, """
out = torch.full((2, 15), 7, dtype=torch.int64, device="cuda")  # both results 8 bytes past a 16-byte boundary
zk.msm_dev(ds, db, out[0, 1:13])
zk.msm_dev(ds[:0], db[:0], out[1, 2:14])
save(out)
""", s, pts, ZKGPU_MSM_HOST_WAIT_US=wait_us)
    assert np.array_equal(got[0, 1:9], oracle.multiexp(s, pts))
    assert np.array_equal(got[0, 9:13], oracle.to_mont(1, oracle.FQ))
    assert not got[1, 2:14].any()
    for row, a, b in ((got[0], 1, 13), (got[1], 2, 14)):
        assert (row[:a] == 7).all() and (row[b:] == 7).all()


def test_answered_where_launches_wait_for_their_kernels(oracle, tmp_path):
    """the slot is watched before its kernel starts: no call sits out the wait"""
    n = 1000
    s, pts = oracle.rand_fr(n, 911), oracle.rand_bases(n, 912)
    got = run_child(tmp_path, """
out = torch.zeros((9, 12), dtype=torch.int64, device="cuda")
ms = []
for row in out:
    t = time.perf_counter()
    zk.msm_dev(ds, db, row)
    torch.cuda.synchronize()
    ms.append(1e3 * (time.perf_counter() - t))
assert sorted(ms)[4] < 150, ms
save(out)
""", s, pts, CUDA_LAUNCH_BLOCKING="1", ZKGPU_MSM_HOST_WAIT_US="300000")
    want = oracle.multiexp(s, pts)
    assert all(np.array_equal(row[:8], want) for row in got)


def test_captured_call_replays_on_new_scalars(oracle, tmp_path):
    """under stream capture the kernel does the last step: a replay sums whatever the buffers hold then"""
    n = 700
    s, pts = oracle.rand_fr(2 * n, 931), oracle.rand_bases(n, 932)
    got = run_child(tmp_path, """
st = torch.cuda.Stream()
cur = ds[:len(db)].clone()
out = torch.zeros(12, dtype=torch.int64, device="cuda")
rows = torch.zeros((3, 12), dtype=torch.int64, device="cuda")
zk.msm_dev(cur, db, out, stream=st)
torch.cuda.synchronize()
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph, stream=st):
    zk.msm_dev(cur, db, out, stream=st)
for k in range(3):
    cur.copy_(ds[len(db):] if k == 1 else ds[:len(db)])
    torch.cuda.synchronize()
    graph.replay()
    torch.cuda.synchronize()
    rows[k] = out
    out.zero_()
    torch.cuda.synchronize()
save(rows)
""", s, pts)
    want = [oracle.multiexp(np.ascontiguousarray(v), pts) for v in (s[:n], s[n:])]
    assert np.array_equal(got[:, :8], np.stack([want[0], want[1], want[0]]))


@pytest.mark.parametrize("wait_us", ["1", "20", "3000"])
def test_late_answers_and_full_slots(oracle, tmp_path, wait_us):
    """Four threads with a stream each and more calls in flight than there are
    slots.  With a wait of 1 us the kernels give up before the answer and it
    comes late, into slots that are used again; with 20 us it is a race."""
    n, calls = 64, 400
    s, pts = oracle.rand_fr(n + calls, 941), oracle.rand_bases(n, 942)
    got = run_child(tmp_path, """
n = len(db)
calls = len(ds) - n
out = torch.zeros((calls, 12), dtype=torch.int64, device="cuda")
streams = [torch.cuda.Stream() for _ in range(4)]
errors = []
def work(t):
    try:
        for i in range(t, calls, 4):
            zk.msm_dev(ds[i:i + n], db, out[i], stream=streams[t])
    except Exception as e:
        errors.append(e)
torch.cuda.synchronize()
threads = [threading.Thread(target=work, args=(t,)) for t in range(4)]
for t in threads: t.start()
for t in threads: t.join()
assert not errors, errors
torch.cuda.synchronize()
save(out)
""", s, pts, ZKGPU_MSM_HOST_WAIT_US=wait_us)
    for i in range(calls):
        assert np.array_equal(got[i, :8], oracle.multiexp(np.ascontiguousarray(s[i:i + n]), pts)), i
