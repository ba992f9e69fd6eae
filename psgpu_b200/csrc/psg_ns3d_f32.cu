// psg_ns3d_f32.cu -- FP32 3D engine of one grid size, PSG_GRID (compiled once per size, so that
// the sizes build in parallel).
#include "psg_ns3d_impl.cuh"
template <>
psg::Engine3DBase* psg::make_engine3d<float, PSG_GRID>() { return new psg::Engine3D<float, PSG_GRID>(); }
