"""The bench line's roofline on the CPU: profiled counters stand for one launch over the whole workload, so
they are used for that alone; an AUTO call is named after the plan that takes as long."""
import bench


def test_profiled_counters_only_for_the_captured_workload():
    n = bench.WORKLOAD["n_cand"]
    dram, moved = bench.profiled("pair_lane_kernel", n, 1)
    assert dram == 182574080 and moved == 2056652380 * 128
    assert bench.profiled("pair_lane_kernel", n, 8) == (None, None)          # a rank's slice of the transactions
    assert bench.profiled("pair_lane_kernel", n // 2, 1) == (None, None)     # another number of candidates
    assert bench.profiled("cand_stream_kernel", n, 1) == (None, None)        # no capture
    assert bench.profiled("k1_lane_tm_kernel", n, 1) == (158003712, None)    # a capture without wavefronts


def test_auto_is_named_after_the_plan_that_takes_as_long():
    class Eng:
        ms = {"pair": 13.2, "lane_tm": 22.1, "stream": 31.0}

        def set_support_plan(self, plan):
            self.plan = plan

        def phase_stats(self, reset=False):
            return {"count_ms": self.ms[self.plan]}

    class torch:
        class cuda:
            synchronize = staticmethod(lambda: None)
    for ms, want in ((13.4, "pair"), (22.3, "lane_tm"), (29.0, "stream")):
        eng = Eng()
        assert bench.dispatched(eng, lambda: None, torch, ms) == want
        assert eng.plan == "auto"
