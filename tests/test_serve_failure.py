"""CPU test of the server's failure path: the runtime (a fake without a
device) reports an error when a completion is looked for, on a lane and on a
batch.  The requests end with FQ_ERR_CUDA, later ones as well, and the server
can still be destroyed."""
import pytest

import fake_cuda

CODE = """
import time
srv = fq.Server(0, 1e9, lanes=2)
fake.fake_event_query({status})
def results(n):
    out, t0 = [], time.monotonic()
    while len(out) < n and time.monotonic() - t0 < 20:
        buf, k = (fq._Result * 16)(), ctypes.c_int()
        fq.lib().fq_server_poll(srv.handle, buf, 16, ctypes.byref(k), 50)
        out += [(r.ticket, r.status, r.energy) for r in buf[:k.value]]
    return sorted(out)
for _ in range(2):
    tickets = [srv.submit(n, graph(n), [0.1, 0.2], [0.3, 0.4]) for n in {sizes}]
    done = results(len(tickets))
    assert [d[0] for d in done] == tickets, (done, tickets)
    assert all(d[1:] == (fq.ERR_CUDA, 0.0) for d in done), done
assert srv.stats()["pending"] == 0
srv.close()
print("closed")
"""


@pytest.mark.parametrize("sizes", [[17, 20], [9, 12, 14], [10, 18]])
def test_failed_completions_are_reported(tmp_path, sizes):
    out = fake_cuda.run(CODE.format(status=719, sizes=sizes), tmp_path)
    assert "closed" in out
