"""The package calls torch through its public names only."""
import glob
import os
import re

import fastlpr_b200


def test_no_private_torch_names():
    for path in glob.glob(os.path.join(os.path.dirname(fastlpr_b200.__file__), "*.py")):
        with open(path) as f:
            found = re.findall(r"torch(?:\.[a-z]\w*)*\._[A-Za-z]\w*", f.read())
        assert not found, (os.path.basename(path), found)
