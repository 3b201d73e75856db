"""Threads that stage host matrices for different GPUs do not wait for each other; for one GPU they take turns."""
import threading

import numpy as np

from scalingelections_b200 import api


def test_devices_stage_side_by_side(monkeypatch):
    inside = {"cpu": threading.Event(), "meta": threading.Event()}
    leave = threading.Event()

    def stub(src, out, n, dev, *rest):
        inside[str(dev)].set()
        if str(dev) == "cpu":
            assert leave.wait(30)

    monkeypatch.setattr(api, "_stage_locked", stub)
    a = np.zeros(16, dtype=np.uint32)
    threads = [threading.Thread(target=api._stage_to_device, args=(a, "cpu"))]
    threads[0].start()
    assert inside["cpu"].wait(30)
    threads.append(threading.Thread(target=api._stage_to_device, args=(a, "meta")))
    threads[1].start()
    side_by_side = inside["meta"].wait(5)
    inside["cpu"].clear()
    threads.append(threading.Thread(target=api._stage_to_device, args=(a, "cpu")))
    threads[2].start()
    in_turn = not inside["cpu"].wait(0.5)
    leave.set()
    for t in threads:
        t.join()
    assert side_by_side and in_turn
