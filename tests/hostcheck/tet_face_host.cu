// Host-side instantiation of the tetrahedron face configuration for the CPU tests.
#include "../../modfem_gb300/csrc/dg_face.cuh"

using namespace gbfem;

extern "C" int host_tet_face_config(const unsigned char *lo, const unsigned char *ln) { return tet_face_config(lo, ln); }
