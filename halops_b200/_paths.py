"""Where the build puts what the package loads.  Standard library only."""

import os
import sysconfig

LIB_DIR = os.path.join(os.path.dirname(os.path.abspath(__file__)), "lib")


def fast_path_file(torch_version: str) -> str:
    """The module of csrc/fast_path.cpp reads the fields of torch's C++ objects and of CPython's, so it
    serves the versions it was compiled against and no others: both are in its name."""
    return os.path.join(LIB_DIR, f"halops_b200_fast_path.{sysconfig.get_config_var('SOABI')}.torch-{torch_version}.so")
