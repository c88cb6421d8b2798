"""The library's reused host blocks. Across a fork: a child made while other threads take and give back
blocks can do so too (it frees the arrays that it inherited). A child that does not end is killed and
counted."""

import os
import random
import threading
import time
import warnings

from unround import native

FORKS = 400


def _ends(child: int, seconds: float = 5.0) -> bool:
    end = time.monotonic() + seconds
    while time.monotonic() < end:
        if os.waitpid(child, os.WNOHANG)[0] == child:
            return True
        time.sleep(0.001)
    os.kill(child, 9)
    os.waitpid(child, 0)
    return False


def test_children_made_while_blocks_are_taken():
    library = native._library()
    take, give = library.unround_b200_host_block, library.unround_b200_host_block_free
    done = threading.Event()

    # Thousands of idle blocks up to the limit, so that a block given back looks through them for the
    # oldest (their pages are never touched).
    held = [take(490_000) for _ in range(4500)]
    for block in held:
        give(block)

    def work(seed: int) -> None:
        rng = random.Random(seed)
        while not done.is_set():
            some = [take(int(2.0 ** rng.uniform(20, 26))) for _ in range(6)]
            for block in some:
                give(block)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for thread in threads:
        thread.start()
    hung = 0
    try:
        with warnings.catch_warnings():
            warnings.simplefilter("ignore", DeprecationWarning)
            for _ in range(FORKS):
                child = os.fork()
                if child == 0:
                    give(take(5000))
                    os._exit(0)
                hung += not _ends(child)
                if hung > 2:
                    break
    finally:
        done.set()
        for thread in threads:
            thread.join()
    assert hung == 0


def test_a_size_that_cannot_be_had_gives_none():
    library = native._library()
    assert not library.unround_b200_host_block(2**64 - 1)
    assert not library.unround_b200_host_block(2**64 - 64)
