"""Where the library's memory comes from and goes back to (memory.h), as far as that can be seen without a GPU."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "genn_b200", "csrc")


def test_what_goes_back_to_the_pool_came_from_it():
    """A member of the runner that cudaMalloc fills is not handed to poolFree (a stream-ordered free), nor the other way round;
    the near-synapse table has both kinds and says which it is."""
    text = open(os.path.join(CSRC, "runner.cu")).read()

    def members(call):
        return {m.split("->")[-1].split("[")[0] for m in re.findall(call + r"\(&?((?:r->)?\w+(?:\[\w+\])?)", text)} - {"p"}       # (a local)

    assert members("cudaMalloc") & members("poolFree") <= {"nearTable"}
    assert members("poolAlloc") & members("cudaFree") <= {"nearTable"}
    assert "nearExported" in text[text.index("void freeNearTable"):text.index("void dropNear")]
