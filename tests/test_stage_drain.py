"""Index model of xC's bulk-copy ring: a warp whose wait ran out leaves only after it has waited
for every copy it has in flight."""
import pytest


@pytest.mark.parametrize("stages", [2, 3])
@pytest.mark.parametrize("rows", [1, 2, 3, 4, 7])
def test_every_copy_in_flight_is_waited_for(stages, rows):
    for fails_at in range(rows):
        issued = [(r % stages, r // stages & 1) for r in range(min(stages - 1, rows))]
        for it in range(fails_at + 1):
            nxt = it + stages - 1
            if nxt < rows:
                issued.append(((it + stages - 1) % stages, nxt // stages & 1))
            if it < fails_at:   # this row's wait succeeded
                issued.remove((it % stages, it // stages & 1))
        drained = [((fails_at + q) % stages, (fails_at + q) // stages & 1) for q in range(stages) if fails_at + q < rows]
        assert sorted(drained) == sorted(issued)
