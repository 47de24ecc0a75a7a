"""Round counts of many apps on one runtime, more than it has mapped words for: each
app reads its own, words of destroyed apps are taken again, and a new app starts at
zero, also when the one before it was destroyed with its run in flight on a caller's
stream."""
import pytest
import torch

from gpu_workgroup_managment_gb300 import PersistentApp, Runtime, graphs

pytestmark = pytest.mark.gpu


def test_rounds_of_more_apps_than_words():
    paths = [graphs.grid(1, 2 + i % 7) for i in range(300)]
    with Runtime() as r:
        apps = [PersistentApp(r, "lonestar_bfs", g) for g in paths]
        assert all(a.rounds() == 0 for a in apps[:250])
        first = [a.run().rounds for a in apps]
        assert [a.rounds() for a in apps] == first
        # the count of a path's levels grows by one with every vertex
        assert first[:7] == list(range(first[0], first[0] + 7)) and first[:7] * 42 == first[:294]
        for a in apps[::2]:
            a.close()
        again = [PersistentApp(r, "lonestar_bfs", g) for g in paths[:100]]
        assert all(a.rounds() == 0 for a in again)
        assert [a.run().rounds for a in again] == first[:100]
        assert [a.rounds() for a in apps[1::2]] == first[1::2]
        for a in apps + again:
            a.close()


def test_rounds_word_of_an_app_destroyed_in_flight():
    g = graphs.grid(250, 260)
    small = graphs.grid(1, 3)
    stream = torch.cuda.Stream()
    with Runtime() as r:
        with PersistentApp(r, "lonestar_bfs", small) as a:
            want = a.run().rounds
        for _ in range(5):
            a = PersistentApp(r, "lonestar_bfs", g)
            for _ in range(20):
                a.launch(stream=stream.cuda_stream)
            a.close()
            with PersistentApp(r, "lonestar_bfs", small) as b:
                assert b.rounds() == 0
                assert b.run().rounds == want
                stream.synchronize()
                assert b.rounds() == want
