"""The oracle's extended-precision (long double) entry points: what the errors of 64-bit results are taken from."""
import ctypes as C

import numpy as np

import oracle_api as O


def gravity(data, r):
    """Accelerations at Earth-fixed positions r [n, 3] as (hi, lo), hi + lo the value."""
    r = O.f64(r)
    hi, lo = np.zeros_like(r), np.zeros_like(r)
    fn = O.lib().or_gravity_ld
    fn.restype, fn.argtypes = None, [C.c_void_p, C.c_int64] + [C.c_void_p] * 3
    fn(data.h, r.shape[0], O.ptr(r), O.ptr(hi), O.ptr(lo))
    return hi, lo


def stm(data, start, h, steps, r, v, ncorr=7):
    """State transition matrices [n, 6, 6] of the propagation with ncorr passes, by central differences."""
    r, v = O.f64(r), O.f64(v)
    phi = np.zeros((r.shape[0], 6, 6))
    fn = O.lib().or_stm_ld
    fn.restype = None
    fn.argtypes = [C.c_void_p, C.POINTER(O.OrTime), C.c_double, C.c_int32, C.c_int32, C.c_int64] + [C.c_void_p] * 3
    fn(data.h, C.byref(O.tstruct(start)), h, steps, ncorr, r.shape[0], O.ptr(r), O.ptr(v), O.ptr(phi))
    return phi


def propagate(data, start, h, steps, r, v, ncorr=7):
    """Final positions and velocities [n, 3] of the propagation with ncorr passes, rounded to double."""
    r, v = O.f64(r), O.f64(v)
    rf, vf = np.zeros_like(r), np.zeros_like(r)
    fn = O.lib().or_propagate_ld
    fn.restype = None
    fn.argtypes = [C.c_void_p, C.POINTER(O.OrTime), C.c_double, C.c_int32, C.c_int32, C.c_int64] + [C.c_void_p] * 4
    fn(data.h, C.byref(O.tstruct(start)), h, steps, ncorr, r.shape[0], O.ptr(r), O.ptr(v), O.ptr(rf), O.ptr(vf))
    return rf, vf
