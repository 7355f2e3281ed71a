"""A launch leaves nothing behind for the next one or for another host thread: neither how many CTAs the GPU may hold
nor how much shared memory a kernel may use depends on the sizes of other calls."""
import subprocess
import sys
import threading
from pathlib import Path

import pytest
import torch

from photonic_engines_b200.clifford.kernels import chain

pytestmark = pytest.mark.gpu

# One process, so that the first call is the first: a call over many modes, one over few, and the first again.
_TIMES = """
import time, torch
from photonic_engines_b200.clifford import sample_chains
def call(n, m, S):
    g = torch.Generator(device="cuda").manual_seed(m)
    U = torch.zeros(m, m, dtype=torch.complex128, device="cuda")
    U[:, :n] = torch.view_as_complex(torch.randn(m, n, 2, generator=g, dtype=torch.float64, device="cuda")) / m ** 0.5
    s = torch.argsort(torch.rand(S, n, generator=g, device="cuda"), dim=1)
    u = torch.rand(S, n, generator=g, dtype=torch.float64, device="cuda")
    best = 1e9
    for _ in range(6):
        torch.cuda.synchronize()
        t = time.perf_counter()
        sample_chains(U, list(range(n)), s, uniforms=u, mode="cta")
        torch.cuda.synchronize()
        best = min(best, time.perf_counter() - t)
    return best
many, few = (18, 5000, 2000), (18, 300, 2000)
first = call(*many); first_few = call(*few); again = call(*many); again_few = call(*few)
print(first, again, first_few, again_few)
"""


def test_a_call_takes_the_same_time_after_a_call_of_another_size():
    """Occupancy lowered by the call before would cost 1.3 to 1.5 times the time; the runs differ by about 2 %."""
    out = subprocess.run([sys.executable, "-c", _TIMES], capture_output=True, text=True, timeout=300,
                         cwd=Path(__file__).resolve().parent.parent)
    assert out.returncode == 0, out.stderr
    first, again, first_few, again_few = (float(x) for x in out.stdout.split())
    assert again < 1.2 * first
    assert again_few < 1.2 * first_few


def test_two_threads_with_different_mode_counts():
    """Launches of one kernel from two host threads, 0.3 and 78 KB of draw weights: neither is refused, and the rows are
    those of a call alone."""
    dev = torch.device("cuda", torch.cuda.current_device())
    work, rows, errors = [], {}, []
    for m in (40, 10000):
        g = torch.Generator(device=dev).manual_seed(m)
        U = torch.zeros(m, 2, dtype=torch.complex128, device=dev)
        U[:, :2] = torch.view_as_complex(torch.randn(m, 2, 2, generator=g, dtype=torch.float64, device=dev))
        acol, off, mm, nn = U.t().contiguous()[None], *(torch.tensor([x], dtype=t, device=dev) for x, t in
                                                        ((0, torch.int64), (m, torch.int32), (2, torch.int32)))
        S = 8
        args = (acol, off, mm, nn, torch.zeros(S, dtype=torch.int64, device=dev),
                torch.arange(2, device=dev).expand(S, -1).contiguous())
        kw = dict(m_max=m, uniforms=torch.rand(S, 2, generator=g, dtype=torch.float64, device=dev), want_occ=False,
                  mode="cta")
        rows[m] = chain(*args, **kw)[0].cpu()
        work.append((m, args, kw))
    torch.cuda.synchronize()

    def run(m, args, kw):
        try:
            with torch.cuda.stream(torch.cuda.Stream(dev)):
                for _ in range(1000):
                    out = chain(*args, **kw, check_status=False)[0]
                assert torch.equal(out.cpu(), rows[m])
        except Exception as e:                                   # noqa: BLE001 (reported by the main thread)
            errors.append(f"m = {m}: {e}")

    threads = [threading.Thread(target=run, args=w) for w in work]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors


def test_only_variants_with_the_pair_sweep_set_its_tables_aside():
    """FP64 CTAs of one warp, bound by shared memory: two-thread lanes at 16 columns have no pair sweep, one-thread lanes
    do, and their 16.5 KB of tables cost them a CTA per SM (38 KB of layout: five without, four with)."""
    from photonic_engines_b200 import _native as N
    L = N.load()
    with_tables, without = (L.pe_split_slots(N.PRECISIONS["f64"], 16, 32, tpl) for tpl in (1, 2))
    assert 0 < with_tables < without
