"""What the library launches depends on its arguments, not on the process's environment."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pic_b200", "csrc")


@pytest.mark.parametrize("name", sorted(os.listdir(CSRC)))
def test_source_reads_no_environment_variable(name):
    with open(os.path.join(CSRC, name)) as f:
        assert not re.search(r"\b(secure_)?getenv\b|\benviron\b", f.read())
