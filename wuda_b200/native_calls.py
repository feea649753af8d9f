"""Where the operators' native call path (csrc/fast_ops.cpp) lies and how it is loaded.

It is built against one interpreter and one torch, whose object layouts it uses, so its file name says which.  Where there is none
for the running pair, or it cannot be loaded, every operator goes through its Python function: the same checks and the same launches,
at 5 to 12 us more host time per call.
"""
import os

HERE = os.path.dirname(os.path.abspath(__file__))


def file_name():
    import sysconfig
    import torch
    return "_fast.%s-torch%s-abi%d.so" % (sysconfig.get_config_var("SOABI"), torch.__version__, torch._C._GLIBCXX_USE_CXX11_ABI)


class Without:
    """Takes no call."""

    def bind(self, handle):
        pass

    def __getattr__(self, name):
        return lambda *arguments: None


def load():
    import importlib.util
    import sys
    import warnings
    path = os.path.join(HERE, file_name())
    try:
        if not os.path.exists(path):
            raise ImportError("%s is missing" % path)
        spec = importlib.util.spec_from_file_location("wuda_b200._fast", path)
        module = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(module)
    except ImportError as e:
        warnings.warn("wuda_b200: the operators' native call path is not there for this interpreter and torch (%s); calls take the "
                      "longer way through Python.  `python -m wuda_b200.build` builds it." % e, RuntimeWarning, stacklevel=2)
        return Without()
    sys.modules["wuda_b200._fast"] = module
    return module
