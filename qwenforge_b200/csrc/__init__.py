from .build import KernelLibraryError, build_all, host_module, library, library_names, prepare

__all__ = ["KernelLibraryError", "build_all", "host_module", "library", "library_names", "prepare"]
