"""The pool of pinned status blocks (rasterizer._HostWords), with pages of ordinary memory: a finalizer may give a block
back while another is being taken, in the same thread, and blocks are neither lost nor handed out twice."""
import threading

import torch

from photara_drender_gb300 import rasterizer as R


def page_of_ordinary_memory(monkeypatch, before=lambda: None):
    zeros = torch.zeros

    def page(shape, dtype=None, pin_memory=False):
        before()
        return zeros(shape, dtype=dtype)

    monkeypatch.setattr(torch, "zeros", page)


def test_give_while_a_page_is_made(monkeypatch):
    pool, block = R._HostWords(), torch.ones(3)
    page_of_ordinary_memory(monkeypatch, lambda: pool.give(block))
    taken = []
    t = threading.Thread(target=lambda: taken.append(pool.take()), daemon=True)
    t.start()
    t.join(20)
    assert not t.is_alive() and len(taken) == 1
    assert any(b is block for b in (*taken, *pool._free)) and len(pool._free) == 128


def test_blocks_are_handed_out_once(monkeypatch):
    page_of_ordinary_memory(monkeypatch)
    pool, held = R._HostWords(), [[] for _ in range(8)]

    def work(mine):
        for k in range(300):
            mine.append(pool.take())
            if k % 3 == 2:
                pool.give(mine.pop(0))

    threads = [threading.Thread(target=work, args=(h,)) for h in held]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    addresses = [b.data_ptr() for h in held for b in h] + [b.data_ptr() for b in pool._free]
    assert len(addresses) == len(set(addresses)) and sum(map(len, held)) == 8 * 200
