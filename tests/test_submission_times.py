"""A submission's device time: both ends are taken on one stream, it is read while a submission by itself is waited for, and no event
is recorded on two streams. The moments between cannot be arranged from outside, so this reads the source."""
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
RUNTIME = open(os.path.join(ROOT, "vyre_b200", "csrc", "host", "runtime.cu"), encoding="utf-8").read()


def body(name):
    m = re.search(r"\n *(?:int32_t|void|bool|TimePoint\*) " + name + r"\([^)]*\) \{", RUNTIME)
    indent = RUNTIME[m.start() + 1 : m.end()].index(RUNTIME[m.start() + 1 : m.end()].lstrip())
    return RUNTIME[m.end() : RUNTIME.index("\n" + " " * indent + "}", m.end())]


def test_start_and_end_are_taken_on_one_stream():
    s = body("vyb_submit")
    shared = s.index("sub->start = inst->tail->end;")
    assert "if (queued && inst->tail->beside) {" in s[:shared]
    wait = s.index("if (queued) cudaStreamWaitEvent(inst->clock, inst->tail->done, 0);")
    start = s.index("cudaEventRecord(sub->start->event, queued ? inst->clock : inst->stream);")
    assert shared < wait < start < s.index("dispatch(inst, slot_ptr, inst->stream)")
    assert "if (!queued) cudaEventRecord(sub->end->event, inst->stream);" in s and "cudaEventRecord(sub->end->event, inst->clock);" in s


def test_times_that_are_there_are_read_when_the_submission_is_waited_for():
    w = body("vyb_submission_wait")
    # in a chain they are read when they are asked for: an end beside the stream is still on its way
    assert "if (e == cudaSuccess && !s->beside && inst->tail == s) timed = inst->read_times(s->start, s->end, &ns);" in w
    assert w.index("read_times") < w.index("inst->tail = nullptr;")
    g = body("vyb_completion_device_ns")
    assert "if (!c->has_device_ns && c->start) {" in g and g.index("cudaEventSynchronize(c->end->event)") < g.index("read_times") and "std::lock_guard" in g


def test_an_event_is_recorded_on_one_stream_alone():
    """A record that is still to come is not overtaken by the event's next one."""
    assert "time_points[t->beside].push_back(t)" in body("release_time")
    a = body("acquire_time")
    assert "t->beside = beside;" in a and "time_points[beside].back()" in a
    s = body("vyb_submit")
    assert "sub->end = inst->acquire_time(queued);" in s and "sub->start = inst->acquire_time(queued);" in s
    records = re.findall(r"cudaEventRecord\((sub->(?:start|end)->event), ([^)]*)\)", RUNTIME)
    assert records == [("sub->start->event", "queued ? inst->clock : inst->stream"), ("sub->end->event", "inst->stream"), ("sub->end->event", "inst->clock")]
