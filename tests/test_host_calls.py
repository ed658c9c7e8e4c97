"""What the library's host code asks of the CUDA runtime, with the runtime of
tests/fake_cudart.c in front of it: no GPU, no kernel runs."""
from tests.fake_runtime import run

VISCOUS = """
c = cases.boundary_layer_block(4, 6, 3, dy0=1e-3, growth=1.3, viscous=1, precision="ref", solver="sgs")
c.params.flux = FLUX
g = FlowPsi(c.mesh, c.params)
st = c.initial_state(g.geometry()["cellcenter"])
p = g.params
def viscous(v):
    p.viscous = v
    g.set_params(p)
def since(n, pattern):
    return [c.name for c in calls[n:] if c.what == "launch" and pattern in c.name]
"""


def test_viscosities_of_an_older_state_are_made_again():
    """the cells' viscosities are kept per state: an inviscid residual (here
    with the flux that keeps its gradient records) leaves them behind"""
    run(VISCOUS.replace("FLUX", "3") + """
g.set_state(*st); g.residual()
n = len(calls); g.assemble()
assert not since(n, "k_material")        # the residual's own
viscous(0); g.residual()
viscous(1); n = len(calls); g.assemble()
assert len(since(n, "k_material")) == 1  # not the first residual's
n = len(calls); g.assemble()
assert not since(n, "k_material")
p.mu_a1 *= 1.5; g.set_params(p); n = len(calls); g.assemble()
assert len(since(n, "k_material")) == 1  # other constants
""")


def test_viscosities_follow_the_constants_of_the_gradient_records():
    """records made on request fill the viscosities with the constants then in
    force; going back to the earlier constants is a change too"""
    run(VISCOUS.replace("FLUX", "1") + """
g.set_state(*st); g.residual()
viscous(0); g.residual()
viscous(1); a = p.mu_a1; p.mu_a1 = 1.5 * a; g.set_params(p)
g.reconstruction()
p.mu_a1 = a; g.set_params(p); n = len(calls); g.assemble()
assert len(since(n, "k_material")) == 1
""")


def test_gradient_records_of_an_inviscid_residual_are_made_for_viscous_blocks():
    """an inviscid Roe residual writes no gradient records; the viscous face
    Jacobians and the SA system read them"""
    run(VISCOUS.replace("FLUX", "1") + """
g.set_state(*st); g.residual()
n = len(calls); g.assemble()
assert not since(n, "k_grad")            # the residual's own
viscous(0); g.residual()
viscous(1); n = len(calls); g.assemble()
k = [c for c in since(n, "k_grad") + since(n, "k_face_jacobian")]
assert len(k) == 2 and "k_grad" in k[0] and "ILb1E" in k[0], k
n = len(calls); g.assemble()
assert not since(n, "k_grad")
viscous(0); g.residual()
p.viscous = 2; p.turbulence = 1; g.set_params(p); n = len(calls); g.sa_residual()
assert len(since(n, "k_grad")) == 1
""")


def test_face_records_are_made_again_in_new_system_arrays():
    """the flux kernel leaves the compact face Jacobians of an inviscid
    residual; keeping the diagonal blocks or another precision allocates the
    system anew"""
    run("""
c = cases.farfield_cube(4, precision="ref")
g = FlowPsi(c.mesh, c.params)
g.set_state(*c.initial_state(g.geometry()["cellcenter"]))
def made(change):
    g.residual()
    change()
    n = len(calls); g.assemble()
    return len([c for c in calls[n:] if c.what == "launch" and "k_face_jacobian_c" in c.name])
assert made(lambda: None) == 0
assert made(lambda: g.keep_blocks(False)) == 1
assert made(lambda: None) == 0
assert made(lambda: g.keep_blocks(True)) == 1
def mixed():
    p = g.params
    p.precision = 2  # FP32 blocks as before
    g.set_params(p)
assert made(mixed) == 1
""")


def test_a_failed_inference_leaves_the_callers_array_alone():
    """a model wait that gave up (its error bit set by the last layer here)"""
    run("""
from flowpsi_b200 import _native as N
from flowpsi_b200.learned import LearnedStart
c = cases.taylor_green_tets(4, precision="ref")
g = FlowPsi(c.mesh, c.params)
g.set_state(*c.initial_state(g.geometry()["cellcenter"]))
g.residual(); g.assemble()
m = LearnedStart(seed=0)
fail = True
def give_up(c):
    if fail and c.what == "launch" and "k_layer_ws" in c.name:
        args = C.cast(c.args, C.POINTER(C.c_void_p))
        err = C.cast(args[12], C.POINTER(C.c_void_p))[0]  # its last argument, int32_t* err
        C.cast(err, C.POINTER(C.c_int32))[0] = 2
    return 0
on.append(give_up)
x0 = np.full(g.ncells * 5, 7.0)
assert N.lib().fpsi_gnn_predict(m._h, g._ctx, N.dptr(x0)) == -7  # FPSI_E_TIMEOUT
assert (x0 == 7.0).all()
fail = False
assert N.lib().fpsi_gnn_predict(m._h, g._ctx, N.dptr(x0)) == 0
assert not (x0 == 7.0).any()
""")


def test_line_solves_share_one_shared_memory_limit():
    """the limit belongs to the kernel, not to a context: two contexts with
    lines of different lengths, and colours with more and with fewer groups
    than the device has multiprocessors, all launch under one value"""
    run("""
from flowpsi_b200.solver import GeneratedMesh, bc
from tests.test_gpu_line_groups import uneven_lines
limit, need, above = {}, {}, []
def look(c):
    if "k_lsgs_thomas" in c.name:
        if c.what == "attribute":
            limit.setdefault(c.name, set()).add(c.n)
        if c.what == "launch":
            if c.n > min(limit[c.name]):
                above.append(c)
            need.setdefault(c.name, set()).add(c.n)
    return 0
on.append(look)
def solver(n, prec):
    mesh = GeneratedMesh("hex", n=n, bc_side=(0,) * 6, bcs=[bc("farfield")])
    p = cases.farfield_cube(2, precision=prec).params
    p.solver, p.lsgs_max_iter = 1, 2
    g = FlowPsi(mesh, p)
    g.set_state(np.full(g.ncells, 300.0), np.full(g.ncells, 1e5), np.zeros((g.ncells, 3)))
    return g, mesh
def use(g):
    g.residual(); g.assemble(); g.linear_solve()
for prec in ("mixed", "ref", "fp64"):
    a, ma = solver((4, 600, 2), prec)   # too long for shared memory
    a.set_lines(ma.lines_along(1))
    b, mb = solver((110, 2, 110), prec)
    b.set_lines(uneven_lines(mb, 110))
    for s in (a, b, a, b):
        use(s)
    a.close(), b.close()
assert not above, above[0]
assert len(need) == 6 and max(len(v) for v in need.values()) > 1, need
assert all(len(v) == 1 for v in limit.values()), limit
""")


def test_set_up_on_the_default_stream_is_waited_for():
    """the contexts' and models' streams do not wait for the default stream: a
    clear or an upload on it is complete before either stream is given work"""
    run("""
from flowpsi_b200.learned import LearnedStart
pending, early = [], []
def look(c):
    if c.what in ("memset", "copy_up"):
        pending.append(c)
    elif c.what in ("copy_down", "sync_device") or (c.what == "sync" and c.stream <= 1):
        pending.clear()
    elif c.stream > 1 and c.what != "sync" and pending:
        early.append((pending[-1][:6], c[:6]))
        pending.clear()
    return 0
on.append(look)
def step(what):
    assert not early, (what, early[0])

c = cases.boundary_layer_block(4, 6, 3, dy0=1e-3, growth=1.3, viscous=2, precision="ref", sa=True)
g = FlowPsi(c.mesh, c.params)
st = c.initial_state(g.geometry()["cellcenter"])
g.set_state(*st); step("create")
g.residual(); g.set_lines(c.lines); g.assemble(); g.linear_solve(); step("lines")
c = cases.taylor_green_tets(4, precision="ref")
g = FlowPsi(c.mesh, c.params)
g.set_state(*c.initial_state(g.geometry()["cellcenter"]))
p = g.params
p.viscous, p.turbulence = 2, 1
g.set_params(p); g.residual(); step("SA switched on")
p.viscous = p.turbulence = 0; p.solver = 1
g.set_params(p); g.residual(); g.assemble(); g.linear_solve(); step("line solver switched on")
p.solver = 0
g.set_params(p); g.residual(); g.assemble()
m = LearnedStart(seed=0); step("model")
m.predict(g); step("inference")
m.set_params(m.get_params()); m.add_snapshot(g, np.zeros((g.ncells, 5))); m.train(2); step("training")

# the error bits, cleared after a failure
def zero_pivot(c):
    if c.what == "copy_down_async" and c.n == 4:  # of the assembly's error bits
        C.cast(c.q, C.POINTER(C.c_int32))[0] = 1
    return 0
on.append(zero_pivot)
try:
    g.residual(); g.assemble()
    raise SystemExit("no error")
except FpsiError:
    pass
on.remove(zero_pivot)
g.residual(); g.assemble(); step("after a zero pivot")
""")


def test_an_error_is_reported_once():
    """a call that the runtime refused leaves nothing behind that makes the
    next call fail"""
    run("""
c = cases.farfield_cube(4, precision="ref")
g = FlowPsi(c.mesh, c.params)
st = c.initial_state(g.geometry()["cellcenter"])
def refuse(c):
    return 2 if c.what == "copy_up_async" else 0  # cudaErrorMemoryAllocation
on.append(refuse)
try:
    g.set_state(*st)
    raise SystemExit("no error")
except FpsiError:
    pass
on.remove(refuse)
g.set_state(*st)
g.residual()
# nor another context's allocation
def full(c):
    return 2 if c.what == "malloc" else 0
on.append(full)
try:
    FlowPsi(c.mesh, c.params)
    raise SystemExit("no error")
except FpsiError:
    pass
on.remove(full)
g.residual()
""")


def test_a_failed_face_call_waits_for_its_copies():
    """no copy from the caller's arrays is left in flight when a batched face
    call returns an error, whichever of its calls failed"""
    run("""
from flowpsi_b200 import inviscid_riemann_flux, roe_jacobian
from tests.helpers import face_states
faces = face_states(10, 0)
def fail(what, k):
    n = [0]
    def f(c):
        if c.what != what:
            return 0
        n[0] += 1
        return 700 if n[0] == k else 0
    return f
for call in (lambda: inviscid_riemann_flux("roe", *faces), lambda: roe_jacobian(*faces, 1)):
    call()
    for what, k in (("copy_up_async", 2), ("copy_up_async", 4), ("launch", 1), ("copy_down_async", 1)):
        del calls[:]
        on.append(fail(what, k))
        try:
            call()
            raise SystemExit("no error")
        except FpsiError:
            pass
        del on[:]
        ups = [i for i, c in enumerate(calls) if c.what == "copy_up_async"]
        waits = [i for i, c in enumerate(calls) if c.what == "sync" and c.stream == calls[ups[0]].stream]
        assert waits and waits[-1] > ups[-1], (what, k, [c.what for c in calls])
        assert sum(c.what == "malloc_pool" for c in calls) == sum(c.what == "free_pool" for c in calls)
""")


def test_a_failed_call_leaves_no_copy_of_the_callers_arrays_in_flight():
    """each call that moves an array between the caller and the device, with
    each of its copies and launches refused in turn: whatever it queued has
    been waited for when it returns the error"""
    run("""
from flowpsi_b200.learned import LearnedStart
STREAM = ("copy_up_async", "copy_down_async", "copy_async", "launch")
c = cases.taylor_green_tets(4, precision="ref")
c.params.viscous, c.params.turbulence = 2, 1
g = FlowPsi(c.mesh, c.params)
st = c.initial_state(g.geometry()["cellcenter"])
v1, v5 = np.ones(g.ncells), np.zeros((g.ncells, 5))
m = LearnedStart(seed=0)
def ready(sa):
    p = g.params
    p.viscous, p.turbulence = (2, 1) if sa else (0, 0)
    g.set_params(p)
    g.set_state(*st); g.residual(); g.assemble()
tried = 0
for name, sa, f in [
        ("set_state", 1, lambda: g.set_state(*st)), ("get_state", 1, lambda: g.get_state()),
        ("set_eddy_viscosity", 1, lambda: g.set_eddy_viscosity(v1)), ("eddy_viscosity", 1, lambda: g.eddy_viscosity()),
        ("set_nutilde", 1, lambda: g.set_nutilde(v1)), ("nutilde", 1, lambda: g.nutilde()),
        ("residual", 0, lambda: g.residual()), ("dtau", 0, lambda: g.dtau()),
        ("linear_solve", 0, lambda: g.linear_solve(v5)), ("set_iterate", 0, lambda: g.set_iterate(v5)),
        ("get_iterate", 0, lambda: g.get_iterate()), ("predict", 0, lambda: m.predict(g, want=True)),
        ("add_snapshot", 0, lambda: m.add_snapshot(g, v5))]:
    ready(sa)
    f()
    for k in range(1, 100):
        ready(sa)
        del calls[:]
        n = [0]
        def refuse(c):
            n[0] += c.what in STREAM
            return 700 if c.what in STREAM and n[0] == k else 0
        on.append(refuse)
        try:
            f()
            failed = False
        except FpsiError:
            failed = True
        on.remove(refuse)
        if n[0] < k:
            break
        assert failed, (name, k)
        tried += 1
        seen = 0
        for i, c in enumerate(calls):
            seen += c.what in STREAM
            if c.what in ("copy_up_async", "copy_down_async") and seen != k:
                assert any(d.what == "sync" and d.stream == c.stream for d in calls[i:]), (name, k, c)
assert tried > 30, tried
""")


def test_the_reported_device_memory_is_what_is_held():
    """fpsi_info's device_bytes: arrays made on first use and arrays given
    back when options change included"""
    run("""
from flowpsi_b200 import _native as N
from flowpsi_b200.learned import LearnedStart
size = [0]  # what the context has asked for
def look(c):
    if c.what == "malloc":
        size[0] += c.n
    return 0
def reported(g):
    b = C.c_int64()
    N.lib().fpsi_info(g._ctx, None, None, None, C.byref(b))
    return b.value
c = cases.boundary_layer_block(4, 6, 3, dy0=1e-3, growth=1.3, viscous=2, precision="ref", sa=True)
on.append(look)
g = FlowPsi(c.mesh, c.params)
assert reported(g) == size[0]
g.set_state(*c.initial_state(g.geometry()["cellcenter"]))
g.residual(); g.assemble(); g.linear_solve(); g.sa_residual(); g.run(4)
assert reported(g) == size[0]  # the cells' viscosities among it
p = g.params
p.flux, p.viscous, p.turbulence, p.solver = 3, 0, 0, 0
g.set_params(p); g.residual(); g.assemble(); g.linear_solve()
assert reported(g) == size[0]
n0 = reported(g)
g.keep_blocks(False); g.keep_blocks(True)
assert reported(g) == n0       # given back and made again
p.precision = 0
g.set_params(p)
assert n0 < reported(g) < 2 * n0
p.precision = 1
g.set_params(p)
assert reported(g) == n0
g.residual(); g.assemble()
m = LearnedStart(seed=0)
m.predict(g)
assert reported(g) == n0 + 5 * 8 * g.ncells + 4 * (g.ncells + 1) + 4 * 2 * int((c.mesh.arrays().cr >= 0).sum())
""")


def test_a_failed_run_waits_for_the_steps_in_flight():
    """the steps write their norms to pinned memory that the next, longer run
    gives back"""
    run("""
c = cases.farfield_cube(4, precision="ref")
c.params.time_accurate, c.params.newton_iters = 1, 4
g = FlowPsi(c.mesh, c.params)
st = c.initial_state(g.geometry()["cellcenter"])
s = None
for f in (lambda: g.run(6), lambda: g.time_step(), lambda: g.run_timed(6), lambda: g.kernel_times(2)):
    for what, k in (("launch", 5), ("graph", 2)):
        g.set_state(*st)
        del calls[:]
        n = [0]
        def refuse(c):
            n[0] += c.what == what
            return 700 if c.what == what and n[0] == k else 0
        on.append(refuse)
        try:
            f()
            failed = False
        except FpsiError:
            failed = True
        on.remove(refuse)
        if n[0] < k:
            continue  # no graphs in this call
        assert failed, what
        last = max(i for i, c in enumerate(calls) if c.what in ("launch", "graph"))
        stream = calls[last].stream
        assert any(c.what == "sync" and c.stream == stream for c in calls[last:]), (what, [c[:2] for c in calls[last:]])
""")
