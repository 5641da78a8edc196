"""Locations shared by the build script, the ctypes binding and the torch extension."""

import os

PKG_DIR = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(PKG_DIR)
CSRC = os.path.join(PKG_DIR, "csrc")
LIB_DIR = os.path.join(PKG_DIR, "lib")
LIB_PATH = os.path.join(LIB_DIR, "libsigattn_b200.so")
EXT_NAME = "_sigattn_torch"
EXT_PATH = os.path.join(LIB_DIR, EXT_NAME + ".so")
