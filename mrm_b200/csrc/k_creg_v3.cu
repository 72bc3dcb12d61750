// k_creg_v3.cu -- register column kernel of compiled shape 3 (launch.h kCreg).
#define CREG_V 3
#include "k_creg.inc"
