"""oracle/ — CPU restatement of the reference's algorithms for the hot path.

TEST INFRASTRUCTURE ONLY.  Only tests/, __graft_entry__.smoke() and bench.py's
cpu_baseline / --impl reference legs may import this package, and only as the
oracle or the timed CPU baseline — never on the product path
(pipelinerl_b200/ must not import it; tests/test_boundary.py enforces that).

Pinning: the reference (ServiceNow/PipelineRL) ships no tests or golden vectors,
so every function here is pinned against fixtures generated by EXECUTING the
reference
(tests/golden/make_golden.py -> tests/golden/*.npz|json; checked by
tests/test_oracle_golden.py).  Parts with no executable reference here are
marked "parity unpinned" in their own module docstring.
"""
