"""What the library enqueues, where and in which order, and what it does when a call fails: its host side on
the CPU, with a fake of the CUDA runtime (fake_cudart.cpp)."""
import pytest

import fake_cuda


@pytest.fixture(scope="module")
def fake(tmp_path_factory, lib):
    return fake_cuda.compile_fake(tmp_path_factory.mktemp("fake"))


@pytest.mark.parametrize("batch", [False, True])
def test_a_phase_that_could_not_be_enqueued_is_over(fake, batch):
    """A kernel of the first wave fails to launch: the call reports it, nothing of the wave is launched behind
    it, and the calls that follow do not go on with the failed phase."""
    fake_cuda.run(fake, """
        c = runtime.Context(oligo())
        b = runtime.Batch(max_slots=2) if %r else None
        def run():
            if b: b.run(A.PHASE_STELLAR, [(c, [0], 30000, 0, 30000, 1)])
            else: c.run_phase(A.PHASE_STELLAR, [0], 30000)
        sync = b.sync if b else c.sync
        fake.fake_busy(24, 100)                  # ends in the tail pass, after the first look at the counters
        run(); sync()
        assert len(log("tail_kernel")) == 1
        fake.fake_fail(b"trav_kernel", 0)
        try:
            run()
            assert False
        except A.SkirtError as e:
            assert e.code == A.SKG_ERR_CUDA
        kernels = log("launch ")
        assert len(kernels) == 1 and "launch_kernel" in kernels[0], kernels
        sync()
        assert not log("launch ")                # no waves and no tail pass of the failed phase
        run(); sync()
        assert len(log("tail_kernel")) == 1
    """ % batch)


@pytest.mark.parametrize("what,code", [("trav_kernel", "A.SKG_ERR_CUDA"), ("instantiate", "A.SKG_ERR_OOM")])
def test_a_capture_that_failed_is_closed(fake, what, code):
    """A launch fails while a batch is captured, or its graph cannot be made: nothing runs, and the next
    captured run works."""
    fake_cuda.run(fake, """
        c = runtime.Context(oligo())
        b = runtime.Batch(max_slots=2)
        def run(graph):
            b.run(A.PHASE_STELLAR, [(c, [0], 30000, 0, 30000, 1)], graph=graph)
        fake.fake_busy(24, 100)
        run(False); b.sync()
        log()
        fake.fake_fail(b"%s", 0)
        try:
            run(True)
            assert False
        except A.SkirtError as e:
            assert e.code == %s
        assert len(log("uncapture")) == 1
        b.sync()
        assert not log("launch ")
        run(True); b.sync()
        lines = log()
        assert any(l.startswith("replay") for l in lines) and any("end_kernel" in l for l in lines)
    """ % (what, code))


def test_waves_added_to_a_replay_are_launched_as_captured(fake):
    """Between two replays of a captured batch a smaller phase of another kind runs directly: the waves and the
    tail pass added to the second replay have the captured pool and kind of walk.  Budgets frozen in the
    captured launches make another graph."""
    fake_cuda.run(fake, """
        keeps, plain = runtime.Context(oligo(write_absorption=True)), runtime.Context(oligo(write_absorption=False))
        b = runtime.Batch(max_slots=2)
        def run(ctx, n, graph, **kw):
            log()
            b.run(A.PHASE_STELLAR, [(ctx, [0], n, 0, n, 1)], graph=graph, **kw)
            b.sync()
            return log()
        waves = lambda lines: [l for l in lines if "launch " in l and "WaveParams" in l]
        fake.fake_busy(1, 60000)
        run(keeps, 60000, True)
        run(plain, 22000, False, precision=A.PREC_FP64, pool=21000, max_scatt=9, refill=3)
        # more waves than were captured, and the tail pass, behind the replay
        fake.fake_busy(30, 60000)
        lines = run(keeps, 60000, True)
        assert not any(l.startswith("capture") for l in lines)
        added = waves(lines[lines.index("end of replay"):])
        assert len(added) == 40                           # eight waves of five kernels
        replayed = waves(lines[:lines.index("end of replay")])
        what = lambda l: (l.split(" (")[0].split("launch ")[1].split("(")[0], l.split("npool")[1])
        for l in added:
            assert what(l)[1] in {what(r)[1] for r in replayed}, l
            assert what(l)[0] in {what(r)[0] for r in replayed}, l
        run(plain, 22000, False, precision=A.PREC_FP64, pool=21000, max_scatt=9, refill=3)
        fake.fake_busy(24, 100)
        lines = run(keeps, 60000, True)
        tail = [l for l in lines if "tail_kernel" in l]
        assert len(tail) == 1 and "<float" in tail[0] and "npool 65536" in tail[0] and "refill 0" in tail[0], tail
        for kw in (dict(max_scatt=7), dict(refill=5)):
            lines = run(keeps, 60000, True, **kw)
            (k, v), = kw.items()
            assert any(l.startswith("capture") for l in lines)
            assert all("%s %d " % (k, v) in l for l in waves(lines))
    """)


@pytest.mark.parametrize("graph", [False, True])
def test_a_batch_waits_for_its_simulations_resets(fake, graph):
    """Resets are enqueued on the contexts' streams; a batch's launches, on another stream, wait for them, and
    for nothing where the contexts have been synchronised since."""
    fake_cuda.run(fake, """
        ctxs = [runtime.Context(oligo()) for _ in range(3)]
        b = runtime.Batch(max_slots=4)
        run = lambda: b.run(A.PHASE_STELLAR, [(c, [0], 9000, 0, 9000, 1) for c in ctxs], graph=%r)
        run(); b.sync()
        ctxs[2].sync()
        for c in ctxs: c.reset_tallies()
        ctxs[1].sync()
        lines = log()
        # the event behind each context's last memset
        ends = [l.split()[1:] for a, l in zip(lines, lines[1:]) if l.startswith("record") and a.startswith("memset")]
        assert len(ends) == 3 and len({s for _, s in ends}) == 3, ends
        run(); b.sync()
        lines = log()
        first = next(i for i, l in enumerate(lines) if l.startswith(("launch", "replay")))
        stream = lines[first].split()[1]
        waits = [l.split()[1:] for l in lines[:first] if l.startswith("wait")]
        waits = [w for w in waits if w[1] in {e for e, _ in ends}]
        assert waits == [[stream, ends[0][0]], [stream, ends[2][0]]], (waits, ends)
    """ % graph)


@pytest.mark.parametrize("call", ["c.run_phase(A.PHASE_STELLAR, [0], 30000, stream=77)",
                                  "c.read_instrument_device(0, cube.ctypes.data, stream=77)"])
def test_a_callers_stream_waits_for_the_reset(fake, call):
    fake_cuda.run(fake, """
        import numpy as np
        c = runtime.Context(oligo())
        cube = np.zeros(64)
        c.reset_tallies()
        end = [l for l in log() if l.startswith("record")][-1].split()[1]
        %s
        assert "wait 77 " + end in log()
    """ % call)


def test_what_follows_a_phase_on_a_callers_stream_waits_for_its_tail_pass(fake):
    """The tail pass is enqueued when the phase is completed: the context's stream goes on behind it (reads,
    resets, the dust emission), and so does the next phase on yet another stream, which shares its pool."""
    fake_cuda.run(fake, """
        c = runtime.Context(oligo())
        own = [l for l in log("memset")][-1].split()[1]
        fake.fake_busy(24, 100)
        for call in (c.sync, c.reset_tallies, lambda: c.run_phase(A.PHASE_STELLAR, [0], 30000, stream=88)):
            c.run_phase(A.PHASE_STELLAR, [0], 30000, stream=77)
            log()
            call()
            lines = log()
            tail = next(i for i, l in enumerate(lines) if "tail_kernel" in l)
            assert lines[tail].startswith("launch 77 ")
            end = [l for l in lines[tail:] if l.startswith("record") and l.endswith(" 77")][-1].split()[1]
            wait = lines.index("wait %s %s" % (own, end))
            assert not any(l.startswith(("memset", "launch")) for l in lines[tail + 1:wait])
            done = lines[wait + 1].split()
            assert done[0] == "record" and done[2] == own
            if lines[-1].endswith(" 88"):
                first = next(i for i, l in enumerate(lines) if l.startswith(("launch 88", "memset 88")))
                assert "wait 88 " + done[1] in lines[:first]
            c.sync()
    """)


def test_the_next_launch_of_a_batch_waits_for_its_tail_pass(fake):
    fake_cuda.run(fake, """
        c = runtime.Context(oligo())
        b = runtime.Batch(max_slots=2)
        fake.fake_busy(24, 100)
        run = lambda s: b.run(A.PHASE_STELLAR, [(c, [0], 30000, 0, 30000, 1)], stream=s)
        run(77)
        log()
        run(88)
        lines = log()
        tail = next(i for i, l in enumerate(lines) if "tail_kernel" in l)
        end = next(l for l in lines[tail:] if l.startswith("record") and l.endswith(" 77")).split()[1]
        first = next(i for i, l in enumerate(lines) if l.startswith(("launch 88", "memset 88")))
        assert "wait 88 " + end in lines[tail:first]
        b.sync()
    """)


def test_tables_that_can_be_missed_leave_room_for_those_that_cannot(fake):
    """On a device with room for a tree scene's own tables but not for its octant records too, the scene is set
    up and walks on the lattice records; the records are made while a quarter of the device stays free."""
    fake_cuda.run(fake, """
        import numpy as np
        splits = np.zeros(585, dtype=np.uint8)             # every node of levels 0 to 2: 512 leaves
        splits[:73] = 1
        def scene():
            m = models.pan_disk(nlambda=50, npix=8, dust_emission=True, write_absorption=True)
            m.dustGrid = runtime.tree_from_splits(A.GRID_OCTREE, (-1., -1., -1., 1., 1., 1.), splits)
            m.rho = np.full((1, 512), 1e-24)
            return m
        def context(memory):
            fake.fake_memory(memory)
            c = runtime.Context(scene())
            fake.fake_memory(8 << 30)
            log()
            c.run_phase(A.PHASE_STELLAR, [0], 9000); c.sync()
            walks = {l.split("Tree")[1].split("Stepper")[0] for l in log("trav_kernel")}
            need = c.device_bytes
            c.close()
            assert fake.fake_used() == 0
            return need, walks
        os.environ["SKG_TREE_RECORDS"] = "lattice"
        need, walks = context(8 << 30)
        assert walks == {"Lattice"}
        del os.environ["SKG_TREE_RECORDS"]
        full, walks = context(8 << 30)
        assert walks == {"Octant"} and full == need + 256 * 512
        for room in (0, 1000, 256 * 512, need // 4):
            assert context(need + room) == (need, {"Lattice"}), room
        assert context((full + 4096) * 4 // 3) == (full, {"Octant"})
    """)


def test_a_divisor_of_one_hands_over_after_the_first_wave(fake):
    """SKG_TAIL_DIV=1 (the plain path: one thread runs a packet's whole life) leaves one wave before the tail
    pass, and later phases as many waves up front as before."""
    fake_cuda.run(fake, """
        c = runtime.Context(oligo())
        def waves():
            log()
            c.run_phase(A.PHASE_STELLAR, [0], 30000)
            c.sync()
            lines = log("launch ")
            return sum("launch_kernel" in l for l in lines), sum("tail_kernel" in l for l in lines)
        fake.fake_busy(40, 30000)
        before = waves(), waves()
        os.environ["SKG_TAIL_DIV"] = "1"
        assert waves() == (1, 1)
        del os.environ["SKG_TAIL_DIV"]
        assert waves() == before[1]
    """)


def test_absorbed_luminosities_are_read_on_a_full_device(fake):
    """The transpose takes its scratch on the device; without room for it the tables are read all the same."""
    fake_cuda.run(fake, """
        import numpy as np
        c = runtime.Context(oligo(wavelengths=[(0.4 + 0.1 * i) * 1e-6 for i in range(3)], write_absorption=True))
        nc, nl = 6 * 5 * 4, 3
        fake.fake_fill.argtypes = [C.c_size_t]
        fake.fake_fill(8 * nc * nl)                        # the tables, [wavelength][cell]
        fake.fake_memory(fake.fake_used())
        c.dust_tallied = True
        for labs in c.read_absorption():
            assert np.array_equal(labs, np.arange(nc * nl).reshape(nl, nc).T)
        assert not log("cell_major")
        fake.fake_memory(8 << 30)
        c.read_absorption()
        assert len(log("cell_major")) == 2
    """)
