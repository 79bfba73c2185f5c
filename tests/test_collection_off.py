"""Garbage collection stays off until the last of several blocks that turn it off ends, as when one thread serves while another
captures a train step; then it is what it was."""
import gc
import threading

from bats_gb300 import serving, train


def test_blocks_that_overlap():
    assert gc.isenabled()
    first, second = serving.no_gc_pauses(), train.no_collection()
    first.__enter__()
    second.__enter__()
    first.__exit__(None, None, None)
    off_in_second = not gc.isenabled()
    second.__exit__(None, None, None)
    assert off_in_second and gc.isenabled()


def test_blocks_of_many_threads():
    wrong = []

    def run():
        for _ in range(300):
            with train.no_collection():
                if gc.isenabled():
                    wrong.append(1)

    threads = [threading.Thread(target=run) for _ in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong and gc.isenabled()


def test_left_off_when_it_was_off():
    gc.disable()
    try:
        with train.no_collection():
            assert not gc.isenabled()
        assert not gc.isenabled()
    finally:
        gc.enable()
