"""Which pass kernel a Darlin rank asks for."""
import pytest
import torch


@pytest.mark.parametrize("world,tau,first_owned,alone", [(1, 0, 0, True), (1, 0, 1, False), (1, 0, 7, False), (1, 1, 0, False),
                                                        (2, 0, 0, False)])
def test_pass_of_its_own_only_for_a_rank_that_owns_every_column(monkeypatch, world, tau, first_owned, alone):
    """The kernel for a lone rank updates every column of a block. A key range that starts above the data's smallest
    key leaves the columns below it without an owner (their blocks have no owner's parameters at all): such a rank
    takes the general kernel."""
    from parameter_server_b200.models import darlin
    asked = []

    class _Lib:
        @staticmethod
        def psb_darlin_pass(p, stream):
            asked.append(p._obj.row_state)
            return 0

    monkeypatch.setattr(darlin._lib, "lib", lambda: _Lib)
    monkeypatch.setattr(darlin, "stream_ptr", lambda stream=None: None)
    r = darlin.DarlinRank.__new__(darlin.DarlinRank)
    word = torch.zeros(4, dtype=torch.int32)
    r.S, r.R, r.dev, r.n_rows, r.kkt_threshold, r.phase_ns = world, tau + 2, torch.device("cpu"), 5, 1.0, None
    r.shard_col = [first_owned] + [9] * world
    r.status, r._row_state, r._pass_bar = word, None, word
    r._pass_arrays = lambda: (word, word, word)
    r.run_pass([0, 1], 0, tau)
    assert bool(asked[0]) == alone
