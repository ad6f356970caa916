"""CPU tests, over a CUDA runtime without a device, of what calls under
stream capture leave to the graph and what is done at once, and of what runs
where a cooperative launch is refused."""
import fake_cuda

BARRIER = """
ctx = fq.Context(0)
made = log()
st = ctx.state(17)
def circuit():
    log()
    ctx.qaoa_forward(st, graph(17), [0.1, 0.2], [0.3, 0.4], energy=False)
    return log()
# The grid barrier's counter is zeroed with the context, and waited for.
zero = [i for i, x in enumerate(made) if x == "memset"]
assert zero and "sync" in made[zero[-1]:], made
# Captured first, then called: neither run depends on the other's reset.
fake.fake_capture(1)
captured = circuit()
fake.fake_capture(0)
assert [x.split()[0] for x in captured] == ["launch"], captured
assert [x.split()[0] for x in circuit()] == ["launch"]
# A wait that gave up: the counter is reset when the host hears of it, not by
# the next launch, which may be the replay of a captured one.
log()
assert fq.lib().fq_ctx_selftest_wait(ctx.handle) == fq.OK
assert fq.lib().fq_ctx_synchronize(ctx.handle) == fq.ERR_TIMEOUT
reset = log()
assert "memset" in reset and reset[-1] == "sync", reset
print("ok")
"""


def test_barrier_counter_is_ready_at_every_launch(tmp_path):
    assert "ok" in fake_cuda.run(BARRIER, tmp_path)


DEEP = """
ctx = fq.Context(0)
states = {n: ctx.state(n) for n in (2, 9, 12, 15)}
def circuit(n, P):
    log()
    ctx.qaoa_forward(states[n], graph(n), [0.1] * P, [0.3] * P, energy=False)
    return log()
for n, P in ((9, 60), (12, 64), (15, 40), (2, 1000), (15, 2047)):
    called = circuit(n, P)
    fake.fake_capture(1)
    captured = circuit(n, P)
    fake.fake_capture(0)
    assert all(x.startswith("launch ") for x in called), (n, P, called)
    assert [x + " captured" for x in called] == captured, (n, P, captured)
fake.fake_capture(1)
grown = circuit(9, 5000)
fake.fake_capture(0)
assert grown[0] == "malloc" and all(x.endswith(" captured") for x in grown[1:]), grown
ctx.close()
print("ok")
"""


def test_deep_small_circuits_neither_wait_nor_allocate(tmp_path):
    """More layers than the kernel parameters hold: only launches, captured or
    not (but for growth beyond what every context has room for)."""
    assert "ok" in fake_cuda.run(DEEP, tmp_path)


TABLES = """
ctx = fq.Context(0)
st = {n: ctx.state(n) for n in (20, 21, 26)}
def circuit(n, captured=False, seed=1):
    fake.fake_capture(int(captured))
    log()
    ctx.qaoa_forward(st[n], graph(n, seed), [0.1, 0.2], [0.3, 0.4], energy=False)
    fake.fake_capture(0)
    out = log()
    assert all(("captured" in x) == captured for x in out if x != "malloc"), out
    return {"weights": any("k_put" in x or x.startswith("copy") for x in out),
            "tables": any("k_tile_cuts" in x for x in out), "free": "free" in out}
kept = dict(weights=False, tables=False, free=False)
made = dict(weights=True, tables=True, free=False)
assert circuit(20) == made and circuit(20) == kept
assert circuit(20, seed=2) == made
# The weights are in place (as any other call on the graph leaves them), the
# tables are another size's; then the first circuit is captured.
ctx.cost_phase(st[21], 0.1, graph(21), True, 0.5)
assert circuit(21, captured=True) == made
for _ in range(2):
    assert circuit(21) == made  # whether or not the graph has run
assert circuit(21, captured=True) == made
assert circuit(26) == made  # the tables grow, the captured calls keep theirs
assert circuit(26, captured=True) == made
ctx.close()
print("ok")
"""


def test_captured_circuits_carry_weights_and_tables(tmp_path):
    assert "ok" in fake_cuda.run(TABLES, tmp_path)


PARTITION = """
ctx = fq.Context(0)
st, cs = ctx.state(18), ctx.state(18)
def circuit():
    log()
    ctx.qaoa_forward(st, graph(18), [0.1, 0.2], [0.3, 0.4], energy=False)
    return log()
assert [x for x in circuit() if "k_mid" in x]
fake.fake_cooperative(720)  # the launch is too large for what the stream has
for _ in range(2):
    out = circuit()
    assert any("k_pass" in x for x in out) and not any("k_mid" in x for x in out), out
with fq.Context(0) as c:
    c.energy_grad(18, graph(18), [0.1], [0.3], st, cs)
    assert any("k_pass_dual" in x for x in log())
print("ok")
"""


def test_streams_with_few_sms_run_the_passes(tmp_path):
    assert "ok" in fake_cuda.run(PARTITION, tmp_path)
