// prefilter_fwd.cu — the prefiltered forward kernels (k_forward_prefilter and its batched
// form), compiled from prefilter.cu in a translation unit of their own so that their
// root solves can differ from the rest of the library: here the crate's formulas
// (DVG_EXACT_ROOT_SOLVES), without the certified f32 + Newton shortcuts of
// winding_newton.cuh.  At this kernel's 40-register budget the shortcuts cost more than
// they save (mixed 512x512 scene, 2x2 spp: 2.87 ms with them, 2.76 without), while the
// prefiltered interior, with 168 registers, runs faster with the winding one (4x4 spp, before
// the cell lists took most inside tests: 66.9 against 71.8 ms).
#define DVG_EXACT_ROOT_SOLVES 1
#define DVG_PREFILTER_FORWARD 1
#include "prefilter.cu"
