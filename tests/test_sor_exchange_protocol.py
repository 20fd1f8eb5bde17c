"""The exchange schedule of the chip-resident 3D SOR's cluster form
(`sor3d_solve` in flursys_b200/csrc/sor.cu on `ClusterGroup` of
gridreduce.cuh), restated in Python and run under random interleavings of the
blocks and of the asynchronous stores in flight.

Per sweep a block takes the residual of its odd cells (reads the even halo of
the sweep before), forms and sends the next even cells (reads the odd halo),
takes part in a round of the group that also delivers the even faces, forms and
sends the odd cells (reads the even halo of this sweep) and waits for the odd
faces. The checks: every read finds the sweep's values, no phase of an mbarrier
takes part of another's bytes, and the schedule ends. Reads of a pass are
checked at its beginning and at its end, with other blocks running between."""
import random

import pytest

from .test_conv_pipeline_protocol import Bar


def run_schedule(blocks, sweeps, even_buffers, seed):
    rnd = random.Random(seed)
    nbs = [[b for b in (r - 1, r + 1) if 0 <= b < blocks] for r in range(blocks)]
    bar = [[Bar(1), Bar(1)] for _ in range(blocks)]
    fbar = [[Bar(1), Bar(1)] for _ in range(blocks)]
    # halo[r][buffer][from] = (colour, sweep); the set-up filled the first even buffer and the odd one
    halo = [{("even", k): {n: (0, -1) for n in nbs[r]} for k in range(even_buffers)} | {"odd": {n: (1, -1) for n in nbs[r]}}
            for r in range(blocks)]
    flight = []

    def deliver(i):
        kind, to, src, dst, value = flight.pop(i)
        if kind == "part":
            bar[to][dst].complete_tx(1)
        else:
            halo[to][dst][src] = value
            fbar[to][value[0]].complete_tx(1)

    def block(r):
        def check(buf, colour, sweep):
            for n in nbs[r]:
                assert halo[r][buf][n] == (colour, sweep), ("halo", r, n, halo[r][buf][n], (colour, sweep))

        def wait(b, phase):
            while not b.passed(phase & 1):
                yield

        read = ("even", 0)
        for s in range(sweeps + 1):
            arrives = ("even", (s + 1) % even_buffers)
            if s > 0:  # residual of the odd cells
                check(read, 0, s - 1)
                yield
                check(read, 0, s - 1)
            check("odd", 1, s - 1)  # the next even cells
            yield
            if s < sweeps:
                for n in nbs[r]:
                    flight.append(("face", n, r, arrives, (0, s)))
            yield
            check("odd", 1, s - 1)
            for to in range(blocks):  # the round
                flight.append(("part", to, r, s & 1, None))
            bar[r][s & 1].expect_tx(blocks)
            if s < sweeps:
                fbar[r][0].expect_tx(len(nbs[r]))
            yield from wait(bar[r][s & 1], s >> 1)
            if s == sweeps:
                return
            yield from wait(fbar[r][0], s)
            read = arrives
            check(read, 0, s)  # odd cells
            yield
            check(read, 0, s)
            for n in nbs[r]:
                flight.append(("face", n, r, "odd", (1, s)))
            fbar[r][1].expect_tx(len(nbs[r]))
            yield from wait(fbar[r][1], s)

    threads = [block(r) for r in range(blocks)]
    steps = 0
    while threads or flight:
        steps += 1
        assert steps < 400000, "the schedule does not terminate"
        if flight and rnd.random() < 0.4:
            deliver(rnd.randrange(len(flight)))
        elif threads:
            t = rnd.choice(threads)
            try:
                next(t)
            except StopIteration:
                threads.remove(t)


@pytest.mark.parametrize("blocks", [1, 2, 3, 5, 16])
def test_even_halo_in_two_buffers(blocks):
    for sweeps in (1, 2, 7):
        for seed in range(30):
            run_schedule(blocks, sweeps, 2, seed)


def test_one_even_buffer_is_overwritten_while_it_is_read():
    # the mistake the second buffer is there for, in the restated schedule only
    def finds():
        for seed in range(200):
            run_schedule(3, 7, 1, seed)

    with pytest.raises(AssertionError, match="halo"):
        finds()
