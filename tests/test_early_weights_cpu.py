"""The switch that lets a decode step's products read their weights early belongs to the thread that launches them."""
import threading

from ksa_b200.ops import _lib


def _in_thread(fn):
    out = []
    t = threading.Thread(target=lambda: out.append(fn()))
    t.start()
    t.join()
    return out[0]


def _now():
    on = _lib.set_dependent_launch(False)
    _lib.set_dependent_launch(on)
    return on


def test_another_thread_does_not_see_it():
    before = _lib.set_dependent_launch(True)
    try:
        assert _now() and not _in_thread(_now)
        _in_thread(lambda: _lib.set_dependent_launch(False))
        assert _now()
    finally:
        _lib.set_dependent_launch(before)


def test_steps_of_two_threads_leave_it_off_in_every_order():
    """A saves, B saves, A restores, B restores: the order that left a switch of the whole process on."""
    turn = [threading.Event() for _ in range(4)]
    left = {}

    def step(name, start, saved, go, done):
        start.wait(10)
        before = _lib.set_dependent_launch(True)
        saved.set()
        go.wait(10)
        _lib.set_dependent_launch(before)
        left[name] = _now()
        done.set()
    a = threading.Thread(target=step, args=("a", turn[0], turn[1], turn[2], turn[3]))
    b = threading.Thread(target=step, args=("b", turn[1], turn[2], turn[3], threading.Event()))
    a.start(), b.start()
    turn[0].set()
    a.join(20), b.join(20)
    assert left == {"a": False, "b": False} and not _now()
