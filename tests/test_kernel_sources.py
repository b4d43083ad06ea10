"""What the kernels' sources promise the compiler, where a run that happens to come out right shows nothing (no GPU needed)."""
import os
import re

from geneinfer_b200.ops.build import CSRC


def _source(name):
    with open(os.path.join(CSRC, name)) as f:
        return f.read()


def test_the_router_has_one_pointer_to_the_ids_that_it_writes_and_reads():
    """With few tokens the kernel that writes the experts' ids also buckets them: the struct that the bucketing reads them through
    must be the only way to them, and not one that excludes others (``__restrict__``)."""
    text = _source("grouped_product.cu")
    signature = re.search(r"\nroute_kernel\((.*?)\) \{", text, re.S).group(1)
    held = re.search(r"struct RouteAlign \{(.*?)\};", text, re.S).group(1)
    named = set(re.findall(r"\*\s*(\w+)", held))
    assert "ids" in named and "__restrict__" not in held
    written = set(re.findall(r"(?<!const )(?:int|float)\*\s*(?:__restrict__)?\s*(\w+)", signature))
    assert not written & named, "a second way to memory that the bucketing reads or writes"
