"""A submission's device time: both ends are taken on one stream, it is read while the submission is waited for if it is there by then, and an event whose
record may still be to come is not recorded again. The moments between cannot be arranged from outside, so this reads the source."""
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


def test_times_are_read_when_the_submission_is_waited_for():
    w = body("vyb_submission_wait")
    # the newest submission of a chain alone may leave it to its completion: its end is still on the way between the streams
    assert "if (e == cudaSuccess && !(s->beside && inst->tail == s)) timed = inst->read_times(s->start, s->end, &ns);" in w
    assert w.index("read_times") < w.index("inst->tail = nullptr;")
    g = body("vyb_completion_device_ns")
    assert "if (!c->has_device_ns && c->start) {" in g and g.index("cudaEventSynchronize(c->end->event)") < g.index("read_times") and "std::lock_guard" in g


def test_an_event_is_not_recorded_again_before_its_record_is_there():
    assert "(there ? time_points : late_points).push_back(t)" in body("release_time")
    a = body("acquire_time")
    assert "query_event(late_points[i]->event) == cudaSuccess" in a
    # who gives back times without having read them does not know
    assert not re.search(r"release_time\((?!sub->end|start|end)[^,;]+, true\)", RUNTIME) and "c->inst->release_time(c->end, false);" in RUNTIME
