"""Admission in the serving loop counts the integer GEMM's workspace (no GPU)."""
from sparsebackends_b200 import serving
from tests.test_serving import StubServer


class I8StubServer(StubServer):
    def __init__(self, slots, budget):
        super().__init__(slots, budget)
        self.precision = "f64i8"

    def solve(self, req, slot):
        extra = serving.footprint_bytes(req, "f64i8") - serving.footprint_bytes(req)
        with self.lock:
            self.mem += extra
        out = super().solve(req, slot)
        with self.lock:
            self.mem -= extra
        return out


def _requests(chi):
    return [serving.Request(i, 8, 1.0, chi) for i in range(6)]


def test_footprint_by_precision():
    r = _requests(512)[0]
    assert serving.footprint_bytes(r, "f64i8") - serving.footprint_bytes(r) == serving.workspace_bytes(512) > 0
    assert serving.footprint_bytes(r, "tf32x3") == serving.footprint_bytes(r, "f64") == serving.footprint_bytes(r)
    assert serving.workspace_bytes(64) == 0 and serving.footprint_bytes(_requests(64)[0], "f64i8") == \
        serving.footprint_bytes(_requests(64)[0])


def test_admission_leaves_room_for_the_workspace():
    reqs = _requests(512)
    budget = 3 * serving.footprint_bytes(reqs[0]) + serving.workspace_bytes(512)
    srv = I8StubServer(slots=4, budget=budget)
    srv.run(reqs)
    assert srv.peak_mem <= budget
    plain = StubServer(slots=4, budget=budget)
    plain.run(reqs)
    assert plain.peak >= srv.peak


def test_request_over_the_budget_with_its_workspace_is_rejected():
    reqs = _requests(512)[:1]
    srv = I8StubServer(slots=1, budget=serving.footprint_bytes(reqs[0]))
    try:
        srv.run(reqs)
    except ValueError:
        return
    raise AssertionError("expected a ValueError")
