"""Analytic parameter derivatives of the pixelized-PSF (Fourier) path and of
the mixture-of-Gaussians PSF path (blobs of galaxies and point sources), each
behind a torch.autograd.Function.

For each galaxy, tb_galaxy_fft_jac_prep makes seven derivative items on the
geometry of its value item -- position (x, y) through the derivative of the
Lanczos-3 taps, counts (the unit-flux render), the three shape parameters and
the Sersic index through the derivative of the Gaussian-mixture spectrum,
d/dtheta sum_k a_k exp(-2 pi^2 f^T C_k f) = sum_k (da_k - 2 pi^2 a_k
f^T dC_k f) exp(...) -- and tb_fourier_render_deriv renders them through the
same FFT / Lanczos / crop pipeline as the model.  The vector-Jacobian product
(tb_galaxy_fft_vjp) transforms the upstream gradient instead and contracts all
seven derivative spectra with it in frequency space, so backward neither
renders nor stores the Jacobian.

These replace the finite-difference derivatives of Galaxy.getParamDerivatives
and SersicGalaxy.getParamDerivatives (tractor/galaxy.py:137-223,
tractor/sersic.py:402-445) where exact derivatives are wanted.  The seven
parameters are the first seven fields of a GALAXY_SRC record: px, py,
counts, s0, s1, s2 (shape, per shape_type) and sersic_n.
"""
import ctypes
import functools

import numpy as np
import torch

from . import _lib, batch, render

NPARAM = 7
PARAM_NAMES = ('x', 'y', 'counts', 's0', 's1', 's2', 'sersic_n')


class FourierJacobian(object):
    """Derivative items for the galaxies of a FourierGalaxyRenderer (same PSF
    spectra, WCS and profile tables)."""

    def __init__(self, renderer):
        self.r = renderer
        S = batch.COMP_STRIDE
        # items, component amplitudes, variances and coefficients, the
        # product's workspace
        self._scratch = _lib.Scratch(lambda m: (
            7 * m * _lib.FFT_ITEM.itemsize, m * S * 8, m * S * 32, 4 * m * S * 32,
            self._vjp_bytes(m)))

    @staticmethod
    @functools.lru_cache(maxsize=64)
    def _vjp_bytes(n):
        nb = ctypes.c_int64()
        _lib.check(_lib.load().tb_galaxy_fft_vjp_workspace(n, ctypes.byref(nb)),
                   'tb_galaxy_fft_vjp_workspace')
        return nb.value

    def _work(self, n, stream=None):
        """The scratch of the calls for n sources as tensors: items, component
        amplitudes, variances and coefficients, flags, counter + status."""
        P, w = self._scratch, self._scratch.get(n, stream)
        S = batch.COMP_STRIDE
        return (P.view(w, 0, 7 * n * _lib.FFT_ITEM.itemsize, torch.uint8),
                P.view(w, 1, n * S * 8, torch.float64), P.view(w, 2, n * S * 32, torch.float64),
                P.view(w, 3, 4 * n * S * 32, torch.float64), w[3], w[4])

    def _prep(self, srcs, n, mode, col_stride, stream):
        lib = _lib.load()
        _, (items, camp, cvar, dcoef, ws), nbytes, flags, misc, s = self._scratch.get(n, stream)
        rc = lib.tb_galaxy_fft_jac_prep(srcs.data_ptr(), n, ctypes.addressof(self.r.image),
                                        ctypes.addressof(self.r.tables.struct), items, camp, cvar,
                                        dcoef, batch.COMP_STRIDE, mode, col_stride,
                                        flags.data_ptr(), s)
        _lib.check(rc, 'tb_galaxy_fft_jac_prep')
        return items, camp, cvar, dcoef, flags, misc, ws, nbytes[4]

    def jacobian(self, srcs, n, npix, stream=None):
        """float32 (7, npix) device tensor: row j holds d(model)/d(param j)
        of every galaxy, each at its record's out_off (the layout of the
        value patches).  Also returns the prep flags."""
        with _lib.on_stream(stream):
            out = torch.empty(7 * npix, dtype=torch.float32, device=render.device())
        items, camp, cvar, dcoef, flags, misc, _, _ = self._prep(srcs, n, _lib.MOG_STORE, npix,
                                                                 stream)
        render.fourier_render(items, 7 * n, camp, cvar, self.r.spec.data_ptr(), out.data_ptr(),
                              misc.data_ptr() + 16, dcoef_ptr=dcoef, stream=stream)
        return out.view(7, npix), flags, misc[4:8]

    def vjp(self, srcs, n, grad, stream=None):
        """float64 (n, 7): sum over each galaxy's patch of grad * d(model)/
        d(param), grad laid out like the value patches (tb_galaxy_fft_vjp:
        one adjoint transform per galaxy)."""
        with _lib.on_stream(stream):
            dots = torch.zeros(7 * n, dtype=torch.float64, device=render.device())
            grad = grad.contiguous()
        items, camp, cvar, dcoef, flags, misc, ws, nbytes = self._prep(srcs, n, _lib.FFT_DOT, 0,
                                                                       stream)
        rc = _lib.load().tb_galaxy_fft_vjp(items, n, camp, cvar, dcoef, self.r.spec.data_ptr(),
                                           grad.data_ptr(), dots.data_ptr(), ws, nbytes,
                                           misc.data_ptr() + 16, _lib.stream_ptr(stream))
        _lib.check(rc, 'tb_galaxy_fft_vjp')
        return dots.view(n, 7), flags, misc[4:8]


def records_with_params(template, theta):
    """Device GALAXY_SRC records: `template` (uint8 device tensor of records)
    with its first seven fields replaced by theta (n, 7) float64."""
    n = theta.shape[0]
    rec = template.clone()
    rec.view(torch.float64).view(n, _lib.GALAXY_SRC.itemsize // 8)[:, :NPARAM] = theta
    return rec


class RenderGalaxies(torch.autograd.Function):
    """model = RenderGalaxies.apply(theta, renderer, template, npix):
    the galaxies' model patches (float32, the template records' layout) as
    a differentiable function of theta (n, 7) float64 = (x, y, counts, s0,
    s1, s2, n).  Backward is the analytic vector-Jacobian product of
    FourierJacobian.vjp."""

    @staticmethod
    def forward(ctx, theta, renderer, template, npix):
        n = theta.shape[0]
        rec = records_with_params(template, theta.detach())
        out = torch.empty(npix, dtype=torch.float32, device=theta.device)
        flags = renderer.render_device(rec, n, out)
        ctx.renderer = renderer
        ctx.rec = rec
        ctx.n = n
        ctx.mark_non_differentiable(flags)
        return out, flags

    @staticmethod
    def backward(ctx, grad_out, grad_flags):
        jac = getattr(ctx.renderer, '_jacobian', None)
        if jac is None:
            jac = ctx.renderer._jacobian = FourierJacobian(ctx.renderer)
        g, _, _ = jac.vjp(ctx.rec, ctx.n, grad_out.float())
        return g, None, None, None


# ---------------------------------------------------------------------------
# Mixture-of-Gaussians PSF path: blobs of point sources and galaxies
# ---------------------------------------------------------------------------

class BlobModel(object):
    """The model images of a BlobFitter's blobs as a function of their
    parameters (n_src, 9: x, y, flux per band, log r_e, ee1, ee2, Sersic n),
    and the analytic vector-Jacobian product, both from tb_fit_model_vjp
    (FP64 evaluation: the sources' PSF-convolved mixtures over their masks,
    the derivative columns of Galaxy.getParamDerivatives /
    PointSource.getParamDerivatives, tractor/galaxy.py:137-223,
    tractor/pointsource.py:130-241, taken analytically).  The images are laid
    out as the fitter's data (fit.pix_offsets)."""

    def __init__(self, fitter):
        self.f = fitter
        f = fitter
        P = f.blobs_np['P'].astype(np.int64)
        ns = f.blobs_np['n_slices'].astype(np.int64)
        n_src = f.blobs_np['n_src'].astype(np.int64)
        blob_of = np.repeat(np.arange(f.n_blobs), n_src)
        local = np.arange(f.n_src) - (np.cumsum(n_src) - n_src)[blob_of]
        # the place in gbuf of (source, parameter, slice)
        k = np.arange(int(ns.max()))
        idx = (f.blobs_np['g_off'].astype(np.int64)[blob_of, None, None] +
               (local[:, None] * NPAR_FIT + np.arange(NPAR_FIT))[:, :, None] +
               k * P[blob_of, None, None])
        idx = np.where(k < ns[blob_of, None, None], idx, int(f.gbuf.numel()))
        idx = idx.reshape(f.n_src * NPAR_FIT, -1)
        # slot gbuf.numel() reads a zero appended to the slices
        self._idx = torch.from_numpy(idx).to(f.dev)

    def _prep(self, theta):
        f = self.f
        f.trial.copy_(theta.reshape(-1).to(torch.float64))
        f._prep(all_blobs=True)

    def _launch(self, mode, grad=None, model=None):
        f = self.f
        lib = _lib.load()
        _lib.check(lib.tb_fit_model_vjp(f.d_pass_units.data_ptr(), f.d_order.data_ptr(),
                                        len(f.pass_units_np), f.d_blobs.data_ptr(),
                                        f.d_sources.data_ptr(), f.n_src, f.workspace.data_ptr(),
                                        None if grad is None else grad.data_ptr(),
                                        None if model is None else model.data_ptr(),
                                        f.d_tiles.data_ptr(), f.gbuf.data_ptr(), f.n_bands, mode,
                                        f.misc.data_ptr(), f.misc.data_ptr() + 16,
                                        _lib.stream_ptr()), 'tb_fit_model_vjp')
        render.check_status(f.misc[4:8].clone(), 'tb_fit_model_vjp')

    def model(self, theta):
        """float32 (npix,) device tensor of the blobs' model images."""
        self._prep(theta)
        out = torch.zeros(int(self.f.pix_offsets[-1]), dtype=torch.float32, device=self.f.dev)
        self._launch(_lib.FIT_MODEL, model=out)
        return out

    def vjp(self, theta, grad):
        """float64 (n_src, 9): sum over the images of grad * d(model)/d(theta)."""
        self._prep(theta)
        g = grad.contiguous().to(torch.float32)
        self._launch(_lib.FIT_VJP, grad=g)
        ext = torch.cat([self.f.gbuf, torch.zeros(1, dtype=torch.float64, device=self.f.dev)])
        return ext[self._idx].sum(dim=1).view(self.f.n_src, NPAR_FIT)


NPAR_FIT = _lib.FIT_NPAR


class RenderBlobs(torch.autograd.Function):
    """model = RenderBlobs.apply(theta, blob_model): the blobs' model images
    (float32, the fitter's data layout) as a differentiable function of theta
    (n_src, 9) float64; backward is BlobModel.vjp, the analytic
    vector-Jacobian product (no finite differences, no Jacobian in memory)."""

    @staticmethod
    def forward(ctx, theta, blob_model):
        ctx.blob_model = blob_model
        ctx.save_for_backward(theta)
        return blob_model.model(theta.detach())

    @staticmethod
    def backward(ctx, grad_out):
        theta, = ctx.saved_tensors
        return ctx.blob_model.vjp(theta.detach(), grad_out), None
