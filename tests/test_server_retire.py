"""elhl_server_step moves its finished requests from `active` to `finished` one by one and
exchanges the list at the end.  A return in between would leave a request in both: the
caller takes its result, which deletes it, and the next step reads it.  The read-backs that
can fail there are the device's, so the rule is checked on the source."""
import os
import re

API = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dynemol_gb300", "csrc", "elhl_api.cu")


def test_no_return_while_requests_are_in_both_lists():
    text = re.sub(r"//[^\n]*", "", open(API).read())
    step = text[text.index("int elhl_server_step("):]
    step = step[:step.index("\nint elhl_server_poll(")]
    loop = step[step.index("std::vector<ServerRequest *> keep;"):step.index("sv->active.swap(keep);")]
    assert "sv->finished[r->id] = r;" in loop
    assert not re.findall(r"\breturn\b|\bCU_TRY\(|\bbreak\b|\bgoto\b", loop)
