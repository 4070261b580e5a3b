"""Reconstructions, with and without a tape, from several host threads at once, each on a stream of
its own: every call succeeds and gives what it gives alone.  The levels differ in the shared memory
that their sweeps take, and a kernel's limit on it belongs to all threads."""
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu


def test_threads_do_not_disturb_one_another():
    from warp_psr_b200 import clouds, reconstruct, reconstruct_differentiable
    jobs = []
    for n, depth, precision in [(5000, 6, "input"), (20000, 7, "mixed"), (60000, 7, "input"), (3000, 5, "input"),
                                (800, 4, "mixed"), (400, 5, "input")]:
        p, v = (torch.tensor(a, dtype=torch.float32, device="cuda") for a in clouds.sphere(n))
        jobs.append((p, v, dict(depth=depth, full_depth=3, precision=precision)))
    alone = [reconstruct(p, v, **o).field.coefficients.clone() for p, v, o in jobs]
    torch.cuda.synchronize()
    wrong = []

    def work(k):
        stream = torch.cuda.Stream()
        try:
            with torch.cuda.stream(stream):
                for call in range(40):
                    i = (k + call) % len(jobs)
                    p, v, o = jobs[i]
                    if call % 5 == 4:
                        r = reconstruct_differentiable(p.clone().requires_grad_(True), v, **o)
                        r.iso_value.backward()
                        coefficients = r.coefficients.detach()
                    else:
                        coefficients = reconstruct(p, v, **o).field.coefficients
                    stream.synchronize()
                    if not torch.equal(coefficients, alone[i]):
                        wrong.append((k, call, "differs"))
        except Exception as e:
            wrong.append((k, repr(e)))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, wrong
